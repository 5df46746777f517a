"""The CTU search's shared-memory layout, swept on the host over every even
range and chunk height (ctu_layout.cpp, the header the kernel includes)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.skipif(shutil.which("g++") is None, reason="no C++ compiler")
def test_every_access_inside_its_area(tmp_path):
    exe = str(tmp_path / "ctu_layout")
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", os.path.join(ROOT, "xavs2_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "ctu_layout.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
