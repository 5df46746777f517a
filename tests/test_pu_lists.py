"""The layout of PU lists for the search (pu_lists.cpp, the header the library
includes) against its definition, and its cost."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.skipif(shutil.which("g++") is None, reason="no C++ compiler")
def test_same_lists_in_half_the_time(tmp_path):
    """Callers hand in a new list for every picture, so its layout must stay
    well below what sorting and comparing geometries takes (half; it measured a
    quarter)."""
    exe = str(tmp_path / "pu_lists")
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", os.path.join(ROOT, "xavs2_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "pu_lists.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
    ours, plain = map(float, r.stdout.split())
    assert ours < plain / 2, r.stdout
