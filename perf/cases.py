"""The performance cases of the library: what an encoder (or a server of many
encodes) has it do, through the public entry points of `xavs2_gb300`.

Nine kinds of work, over the sizes they meet in use:

* me          batched motion search of one picture: host pictures in
              (planes of every reference built), full search + sub-pel
              refinement of a PU list, results on the host;
* chain       the full-picture chain of one P picture (captured graph): host
              picture in, search, every inter candidate through the TU chain,
              choice, reconstruction back on the host;
* serve       a burst of pictures of several streams through the server;
* tq          the batched dct / quant / dequant / idct chain on device arrays;
* intra       edges from the reconstruction, then the rough mode decision;
* skip        skip / direct candidates against resident sub-pel planes;
* loopfilter  deblocking + SAO of a 4:2:0 picture;
* lookahead   half-resolution picture + MAD maps;
* percall     one block through the per-call table entries on host memory.

Picture sizes are multiples of 8 (an AVS2 encoder pads its coded pictures to
the smallest CU); only the lookahead, which sees source pictures, takes
others.  All results are whole numbers except two sets of doubles (the
rate-distortion costs of `intra` and `skip`: a whole-number distortion plus
lambda times whole-number bits).
"""
import ctypes
import functools
import math

import numpy as np
import torch

import xavs2_gb300 as xg
import xavs2_gb300.synth as synth

QP = 32
SERVE_SIZES = ((640, 360), (1280, 720), (1920, 1080), (3840, 2160))


# ---- cases --------------------------------------------------------------------
def listed():
    return [
        # the headline workload: every PU of the CU quadtree of a 1080p
        # picture, 2 references, the reference's default range, one predictor
        _me("me_1080p_fs64", 1920, 1080, 2, 64, "quadtree", "zero"),
        # the same search when every PU has its own (neighbour / temporal)
        # predictor and so its own search centre, 720p
        _me("me_720p_fs64_predicted", 1280, 720, 2, 64, "quadtree", "moving"),
        # a small picture with a short range: latency and launches
        _me("me_416x240_fs16", 416, 240, 1, 16, "quadtree", "zero"),
        # the P-picture chain at the largest size and reference count
        {"name": "chain_2160p_fs64", "kind": "chain", "w": 3840, "h": 2160, "refs": 4, "range": 64},
        # serving: ten streams of mixed sizes, four pictures each
        {"name": "serve_mix_fs16", "kind": "serve", "n360": 4, "n720": 3, "n1080": 2, "n2160": 1, "range": 16},
        # the TUs of a picture-sized batch, the square shapes
        {"name": "tq_1e6_squares", "kind": "tq", "n": 1000000, "parts": "squares"},
        # the candidate TUs of a few CUs, every shape: latency
        {"name": "tq_777_all", "kind": "tq", "n": 777, "parts": "all"},
        # intra mode decision of a 1080p picture, every level and strip
        {"name": "intra_1080p", "kind": "intra", "w": 1920, "h": 1080, "hadamard": True, "rough": True},
        # skip / direct decision of a 1080p picture, 5 candidates per CU
        {"name": "skip_1080p", "kind": "skip", "w": 1920, "h": 1080, "refs": 2, "per_cu": 5},
        # in-loop filters of a 2160p picture
        {"name": "loopfilter_2160p", "kind": "loopfilter", "w": 3840, "h": 2160, "lcu_level": 6},
        # lookahead of a 2160p source picture
        {"name": "lookahead_2160p", "kind": "lookahead", "w": 3840, "h": 2160},
        # one 16x16 CU's residual coding by the per-call drop-ins
        {"name": "percall_16x16", "kind": "percall", "part": 2, "qp": QP},
    ]


def _me(name, w, h, refs, rng_, layout, predictors, hadamard=True, frac=2, fast=False):
    return {"name": name, "kind": "me", "w": w, "h": h, "refs": refs, "range": rng_, "layout": layout,
            "predictors": predictors, "hadamard": hadamard, "frac": frac, "fast": fast}


def _log_size(rng, lo, hi, step=8):
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return max(lo, min(hi, int(round(v / step)) * step))


def _picture_size(rng, wmax):
    w = _log_size(rng, 256, wmax)
    return w, max(128, int(w * rng.uniform(0.35, 0.75)) // 8 * 8)


def _me_cost(c):
    """Pixel differences of the search, a PU with its own centre (and an odd range) counted without sharing."""
    own = c["predictors"] != "zero" or c["range"] % 2
    return c["w"] * c["h"] * c["refs"] * (2 * c["range"]) ** 2 * ((15 if c["layout"] == "quadtree" else 6) if own else 1)


def draw(rng):
    kind = rng.choice(["me", "me", "me", "chain", "chain", "serve", "tq", "tq", "intra", "skip", "loopfilter", "lookahead",
                       "percall"])
    if kind == "me":
        while True:
            w, h = _picture_size(rng, 1920)
            c = _me(None, w, h, rng.randint(1, 4), rng.choice([7, 8, 16, 16, 24, 32, 48, 64, 64, 96]),
                    rng.choice(["quadtree", "quadtree", "leaf"]), rng.choice(["zero", "zero", "moving"]),
                    hadamard=rng.random() < 0.8, frac=rng.choice([1, 2, 2, 2]), fast=rng.random() < 0.2)
            del c["name"]
            if _me_cost(c) <= 0.9 * _me_cost(listed()[1]):
                return c
    if kind == "chain":
        while True:
            w, h = _picture_size(rng, 3840)
            c = {"kind": kind, "w": w, "h": h, "refs": rng.randint(1, 4), "range": rng.choice([8, 16, 32, 64])}
            if w * h * c["refs"] * (256 + (2 * c["range"]) ** 2) <= 0.9 * 3840 * 2160 * 4 * 16640:
                return c
    if kind == "serve":
        n = [rng.randint(0, 4), rng.randint(0, 3), rng.randint(0, 2)]
        return {"kind": kind, "n360": n[0] + (0 if any(n) else 2), "n720": n[1], "n1080": n[2], "n2160": 0,
                "range": rng.choice([8, 12, 16, 24])}
    if kind == "tq":
        return {"kind": kind, "n": int(math.exp(rng.uniform(math.log(100), math.log(900000)))),
                "parts": rng.choice(["squares", "all", "small"])}
    if kind == "intra":
        w, h = _picture_size(rng, 1912)
        return {"kind": kind, "w": w, "h": h, "hadamard": rng.random() < 0.8, "rough": rng.random() < 0.8}
    if kind == "skip":
        w, h = _picture_size(rng, 1912)
        return {"kind": kind, "w": w, "h": h, "refs": rng.randint(1, 4), "per_cu": rng.randint(2, 7)}
    if kind == "loopfilter":
        w, h = _picture_size(rng, 3832)
        return {"kind": kind, "w": w, "h": h, "lcu_level": rng.choice([4, 5, 6, 6])}
    if kind == "lookahead":
        w, h = _picture_size(rng, 3832)
        return {"kind": kind, "w": w - rng.choice([0, 2, 4, 6]), "h": h - rng.choice([0, 2, 4, 6])}
    return {"kind": kind, "part": rng.choice([0, 1, 3, 4, 15, 16, 19, 20, 23, 24]), "qp": rng.randint(22, 51)}


# ---- content (made on the device, from the seed alone) ---------------------------
_TAPS = ((0, 0, 0, 64, 0, 0, 0, 0), (-1, 4, -10, 57, 19, -7, 3, -1), (-1, 4, -11, 40, 40, -11, 4, -1),
         (-1, 3, -7, 19, 57, -10, 4, -1))


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _blur(x, sigma):
    r = int(4 * sigma + 0.5)
    k = torch.exp(-0.5 * (torch.arange(-r, r + 1, device=x.device, dtype=torch.float32) / sigma) ** 2)
    k = (k / k.sum()).tolist()
    for axis in (0, 1):
        n = x.shape[axis]
        idx = torch.arange(-r, n + r, device=x.device).clamp(0, n - 1)
        p = x.index_select(axis, idx)
        x = sum(k[i] * p.narrow(axis, i, n) for i in range(2 * r + 1))
    return x


def _base_picture(g, w, h, sigma=3.0):
    """Blurred noise rescaled to [16, 235]."""
    x = _blur(torch.randint(0, 256, (h, w), generator=g, device="cuda").float(), sigma)
    return (16 + (x - x.min()) * (219.0 / (x.max() - x.min()))).round()


def _moved(img, mvx, mvy):
    """out(x, y) = img(x + mv / 4), quarter-pel, AVS2 luma taps, edges repeated."""
    h, w = img.shape
    for axis, n, mv in ((1, w, mvx), (0, h, mvy)):
        at = torch.arange(-3, n + 4, device=img.device) + (mv >> 2)
        p = img.index_select(axis, at.clamp(0, n - 1))
        img = sum(t / 64.0 * p.narrow(axis, k, n) for k, t in enumerate(_TAPS[mv & 3]) if t)
    return img


def _next_picture(g, r, prev, motions, max_px):
    """The previous picture moved by one of `motions` vectors per 8x8 block (one: the whole picture), plus noise;
    also the vector of every 8x8 block."""
    h, w = prev.shape
    mvs = r.integers(-4 * max_px, 4 * max_px + 1, (motions, 2))
    labels = torch.randint(0, motions, ((h + 7) // 8, (w + 7) // 8), generator=g, device="cuda")
    lab = labels.repeat_interleave(8, 0).repeat_interleave(8, 1)[:h, :w]
    out = torch.zeros_like(prev)
    for m in range(motions):
        out = torch.where(lab == m, _moved(prev, int(mvs[m, 0]), int(mvs[m, 1])), out)
    out = out + 2.0 * torch.randn((h, w), generator=g, device="cuda")
    return out.round().clamp(0, 255), mvs[labels.cpu().numpy()]


def _sequence(seed, n, w, h, motions, max_px, pan=0):
    g, r = _generator(seed), np.random.default_rng(seed)
    pics, fields = [_base_picture(g, w, h)], []
    for _ in range(n - 1):
        p, f = _next_picture(g, r, _moved(pics[-1], 4 * pan, 0) if pan else pics[-1], motions, max_px)
        pics.append(p)
        fields.append(f)
    return [p.to(torch.uint8) for p in pics], fields


def _host(t):
    """A page-locked host copy (tensor and numpy view)."""
    p = torch.empty(t.shape, dtype=t.dtype).pin_memory()
    p.copy_(t)
    return p, p.numpy()


class _Raw:
    """Device memory that `owner` holds: the tensor over it keeps the owner alive."""

    def __init__(self, ptr, n, kind, owner):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": kind, "data": (ptr, False), "version": 3}


def _device_view(ptr, n, kind, owner):
    return torch.as_tensor(_Raw(ptr, n, kind, owner), device="cuda")


def _P(t):
    return ctypes.c_void_p(t.data_ptr())


def _stream():
    return ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)


def _check(rc, what):
    if rc:
        raise RuntimeError("%s: %d" % (what, rc))


def _lambda_rd():
    return 2.0 ** ((QP - 11) / 4.0) * 0.68


def _params(case):
    return xg.MeParams(case["range"], int(65536.0 * math.sqrt(_lambda_rd()) + 0.5), int(case.get("hadamard", True)),
                       case.get("frac", 2), int(case.get("fast", False)), 0)


# PU and CU lists depend on the sizes alone, like an encoder's own tables
@functools.lru_cache(maxsize=4)
def _quadtree(w, h, refs):
    return xg.frame_pus(w, h, refs)


@functools.lru_cache(maxsize=16)
def _leaves(w, h, refs, split_seed):
    return xg.cu_pus(xg.split_map_cus(w, h, split_seed), w, h, refs)


# ---- prepare --------------------------------------------------------------------
def prepare(case, seed):
    xg.load()
    return {"kind": case["kind"], **globals()["_prepare_" + case["kind"]](case, seed)}


def _prepare_me(case, seed):
    w, h, refs, R = case["w"], case["h"], case["refs"], case["range"]
    pics, fields = _sequence(seed, refs + 1, w, h, 16, max(2, R // 2))
    pus = _quadtree(w, h, refs) if case["layout"] == "quadtree" else _leaves(w, h, refs, 5)[0]
    if case["predictors"] != "zero":
        # the motion at the PU's middle, summed back to its reference, a little off: what a neighbour's or the
        # co-located block's vector predicts
        pus = pus.copy()
        r = np.random.default_rng(seed + 1)
        pw, ph = np.asarray(xg.PU_W)[pus["part"]], np.asarray(xg.PU_H)[pus["part"]]
        cx, cy = (pus["x"] + pw // 2) // 8, (pus["y"] + ph // 2) // 8
        back = np.cumsum(np.stack(fields[::-1]), axis=0)
        mv = back[pus["ref"], cy, cx] + r.integers(-4, 5, (len(pus), 2))
        pus["mvp_x"], pus["mvp_y"] = mv[:, 0], mv[:, 1]
    sess = xg.MeSession(w, h, refs, len(pus))
    sess.set_pus(pus)
    keep = [_host(p) for p in pics[::-1]]            # the current picture, then reference 0, 1, ...
    out, out_np = _host(torch.zeros((len(pus), 5), dtype=torch.int32))
    prm = _params(case)
    for i, (_, p) in enumerate(keep):
        sess.set_picture(i - 1, p)
    sess.autotune(prm, reps=2)
    return {"sess": sess, "pics": [k[1] for k in keep], "keep": keep, "prm": prm, "out": out,
            "out_np": out_np.reshape(-1).view(xg.RESULT_DTYPE)}


def _prepare_chain(case, seed):
    w, h, refs = case["w"], case["h"], case["refs"]
    pics, _ = _sequence(seed, refs + 1, w, h, 2, 4, pan=12)
    pus, cus = _leaves(w, h, refs, 31)
    sess = xg.MeSession(w, h, refs, len(pus))
    sess.set_pus(pus)
    chain = xg.Chain(sess, cus, QP)
    keep = [_host(p) for p in pics[::-1]]
    for i, (_, p) in enumerate(keep):
        _check(xg.load().xavs2gpu_copy_h2d(ctypes.c_void_p(chain.source(i)), xg.ptr(p), p.nbytes), "copy_h2d")
    prm = _params(case)
    chain.run(prm)
    chain.autotune(prm, reps=1)
    chain.capture(prm)
    o = chain.outputs()
    n = int(o.n_cands)
    search = xg.load().xavs2gpu_me_results_device(sess.h)
    views = {k: _device_view(p, m, t, (chain, sess)) for k, p, m, t in (
        ("levels", o.coef, int(o.n_coef), "<i2"), ("nnz", o.nnz, 5 * n, "<i4"),
        ("residual", o.recon_residual, int(o.n_residual), "<i2"), ("cost", o.cand_cost, n, "<i4"),
        ("ssd", o.dist, 2 * n, "<i4"), ("choice", o.choice, 2 * len(cus), "<i4"), ("search", search, 5 * len(pus), "<i4"))}
    recon, recon_np = _host(torch.zeros((h, w), dtype=torch.uint8))
    return {"sess": sess, "chain": chain, "keep": keep, "cur": keep[0][1], "views": views, "recon": recon,
            "recon_np": recon_np, "recon_dev": o.recon}


def _prepare_serve(case, seed):
    cfg = xg.ServerConfig(0, 24 << 20, 64, QP, _params(case), hbm_reserve_bytes=0, batch_pixels_target=12 << 20)
    srv = xg.Server(cfg)
    streams = []
    for k, key in enumerate(("n360", "n720", "n1080", "n2160")):
        w, h = SERVE_SIZES[k]
        for i in range(case[key]):
            pus, cus = _leaves(w, h, 2, 1000 + i % 2)
            sid = srv.open_stream(w, h, pus, cus, ring=8)
            if sid < 0:
                raise RuntimeError("open_stream: %d" % sid)
            pics, _ = _sequence(seed * 64 + len(streams), 4, w, h, 1, 8)
            streams.append((sid, [p.cpu().numpy() for p in pics]))
    for k in (2, 3):                                  # the references the first picture of a pass is searched against
        for sid, pics in streams:
            _check(srv.submit(sid, pics[k]), "submit")
    _collect(srv, 2 * len(streams))
    return {"srv": srv, "streams": streams}


def _collect(srv, n):
    got = []
    while n > 0:
        r = srv.poll(4096, 20)
        got.append(r)
        n -= len(r)
    return np.concatenate(got)


_TQ_PARTS = {"squares": (0, 1, 2, 3, 4), "small": (0, 1, 2, 15, 16, 20, 19), "all": tuple(xg.TU_PARTS)}


def _prepare_tq(case, seed):
    # the shapes in one order, so that the arrays keep their sizes; quantisers, secondary transforms and all-zero
    # blocks from the seed
    n, r = case["n"], np.random.default_rng(seed)
    blocks, nres, ncoef, _ = synth.tq_blocks(n, seed=3, parts=_TQ_PARTS[case["parts"]])
    blocks["qp"] = r.integers(22, 52, n)
    blocks["flags"] = np.where((blocks["part"] == 0) & (r.random(n) < 0.5), 3, 0)
    zero = r.random(n) < 0.1
    return {"n": n, "blocks": torch.from_numpy(blocks.view(np.uint8).copy()).cuda(),
            "res": synth.tq_residual(blocks, zero, nres, seed=seed, device="cuda"),
            "levels": torch.zeros(ncoef, dtype=torch.int16, device="cuda"),
            "recon": torch.zeros(nres, dtype=torch.int16, device="cuda"),
            "nnz": torch.zeros(n, dtype=torch.int32, device="cuda")}


def _prepare_intra(case, seed):
    w, h = case["w"], case["h"]
    g, r = _generator(seed), np.random.default_rng(seed)
    src = _base_picture(g, w, h)
    recon = (src + torch.randint(-3, 4, (h, w), generator=g, device="cuda")).clamp(0, 255).to(torch.uint8)
    blocks, jobs, esize = synth.intra_fill_jobs(synth.intra_level_blocks(w, h), w, h, r, xg.INTRA_BLOCK_DTYPE,
                                                xg.INTRA_EDGE_JOB_DTYPE)
    n = len(blocks)
    prm = xg.IntraParams(math.sqrt(_lambda_rd()), int(case["hadamard"]), int(case["rough"]),
                         synth.INTRA_DIST2, synth.INTRA_DIST1)
    out = torch.zeros(n * xg.INTRA_RESULT_DTYPE.itemsize, dtype=torch.uint8, device="cuda")
    return {"w": w, "h": h, "n": n, "prm": prm, "src": src.to(torch.uint8), "recon": recon, "esize": esize,
            "blocks": torch.from_numpy(blocks.view(np.uint8).copy()).cuda(),
            "jobs": torch.from_numpy(jobs.view(np.uint8).copy()).cuda(),
            "edges": torch.zeros(esize, dtype=torch.uint8, device="cuda"), "out": out}


def _skip_candidates(r, w, h, refs, per_cu, motion=(-12, 0)):
    """Candidates of every aligned CU: one with four quadrant PUs, then single-PU ones around `motion` (a third of
    them from two references), some repeating the one before; header bits 1..12."""
    rects = []
    for lv in (3, 4, 5, 6):
        s = 1 << lv
        y, x = np.meshgrid(np.arange(0, h - s + 1, s), np.arange(0, w - s + 1, s), indexing="ij")
        rects.append(np.stack([x.ravel(), y.ravel(), np.full(x.size, lv)], 1))
    rects = np.concatenate(rects)
    n = len(rects)
    c = np.zeros((n, per_cu), xg.SKIP_CAND_DTYPE)
    c["x"], c["y"], c["size_log2"] = rects[:, :1], rects[:, 1:2], rects[:, 2:]
    c["cu"] = np.arange(n)[:, None]
    c["rate"] = r.integers(1, 13, (n, per_cu))
    c["ref"] = -1
    c["n_pu"] = 1
    c["n_pu"][:, 0] = 4
    c["ref"][:, 0, :, 0] = r.integers(0, refs, (n, 4))
    c["mv"][:, 0, :, 0] = r.integers(-6, 7, (n, 4, 2)) + motion
    c["ref"][:, 1:, 0, 0] = r.integers(0, refs, (n, per_cu - 1))
    c["mv"][:, 1:, 0, 0] = r.integers(-12, 13, (n, per_cu - 1, 2)) + motion
    if refs > 1:
        both = r.random((n, per_cu - 1)) < 0.35
        c["ref"][:, 1:, 0, 1] = np.where(both, r.integers(0, refs, both.shape), -1)
        c["mv"][:, 1:, 0, 1] = np.where(both[..., None], r.integers(-12, 13, both.shape + (2,)) + motion, 0)
    for j in range(3, per_cu):
        again = r.random(n) < 0.3
        for f in ("n_pu", "ref", "mv"):
            c[f][again, j] = c[f][again, j - 1]
    return c.reshape(-1), n


def _prepare_skip(case, seed):
    w, h, refs = case["w"], case["h"], case["refs"]
    pics, _ = _sequence(seed, refs + 1, w, h, 2, 4, pan=3)
    cands, n_cu = _skip_candidates(np.random.default_rng(seed), w, h, refs, case["per_cu"])
    sess = xg.MeSession(w, h, refs, 1)
    torch.cuda.synchronize()                          # the session reads the pictures on its own stream
    for i, p in enumerate(pics[::-1]):
        sess.set_picture_device(i - 1, p.data_ptr(), w)
    torch.cuda.synchronize()
    n = len(cands)
    return {"sess": sess, "n": n, "n_cu": n_cu, "cands": torch.from_numpy(cands.view(np.uint8).copy()).cuda(),
            "dist": torch.zeros(n, dtype=torch.int32, device="cuda"),
            "cost": torch.zeros(n, dtype=torch.float64, device="cuda"),
            "best": torch.zeros(n_cu, dtype=torch.int32, device="cuda")}


def _blocky(g, w, h, amp):
    x = _blur(torch.randint(0, 256, (h, w), generator=g, device="cuda").float(), 2.0)
    x = 40 + (x - x.min()) * (170.0 / (x.max() - x.min()))
    off = torch.randint(-amp, amp + 1, ((h + 7) // 8, (w + 7) // 8), generator=g, device="cuda")
    return (x + off.repeat_interleave(8, 0).repeat_interleave(8, 1)[:h, :w]).round().clamp(0, 255).to(torch.uint8)


def _prepare_loopfilter(case, seed):
    w, h, level = case["w"], case["h"], case["lcu_level"]
    g, r = _generator(seed), np.random.default_rng(seed)
    src = [_blocky(g, w, h, 6), _blocky(g, w // 2, h // 2, 4), _blocky(g, w // 2, h // 2, 4)]
    # edges of 8x8 blocks: none / luma / both, strengths over the range of the AVS2 tables
    n = (w // 8) * (h // 8)
    scus = np.zeros(n, xg.DEBLOCK_SCU_DTYPE)
    scus["type"] = np.asarray([2, 2, 2, 1, 0])[r.integers(0, 5, (n, 2))]
    scus["type"][np.arange(n) % (w // 8) == 0, 0] = 0
    scus["type"][np.arange(n) // (w // 8) == 0, 1] = 0
    scus["flag"] = r.random((n, 2, 2)) < 0.9
    for k in ("alpha", "alpha_c"):
        scus[k] = r.integers(4, 65, (n, 2))
    for k in ("beta", "beta_c"):
        scus[k] = r.integers(1, 28, (n, 2))
    # SAO per LCU and component: off, one of four edge classes, bands
    s = 1 << level
    wl, hl = (w + s - 1) // s, (h + s - 1) // s
    m = wl * hl
    lcus = np.zeros(m, xg.SAO_LCU_DTYPE)
    lx, ly = np.arange(m) % wl, np.arange(m) // wl
    lcus["avail"] = (ly > 0) | ((ly < hl - 1) << 1) | ((lx > 0) << 2) | ((lx < wl - 1) << 3)
    kind = np.where(r.random((m, 3)) < 0.1, -1, r.integers(0, 5, (m, 3)))
    lcus["type"] = kind
    eo = np.stack([r.integers(0, 7, (m, 3)), r.integers(0, 2, (m, 3)), np.zeros((m, 3), np.int64),
                   -r.integers(0, 2, (m, 3)), -r.integers(0, 7, (m, 3))], 2)
    lcus["offset"][:, :, :5] = np.where((kind >= 0)[..., None] & (kind < 4)[..., None], eo, 0)
    at, to = np.nonzero(kind == 4)
    band = r.integers(0, 29, len(at))
    for k in range(4):
        lcus["offset"][at, to, band + k] = r.integers(-7, 8, len(at))
    return {"w": w, "h": h, "level": level, "src": src, "dst": [torch.zeros_like(p) for p in src],
            "scus": torch.from_numpy(scus.view(np.uint8).copy()).cuda(),
            "lcus": torch.from_numpy(lcus.view(np.uint8).copy()).cuda()}


def _maps(w, h):
    return [-(-w // s) * -(-h // s) for s in (16, 32, 64)]


def _prepare_lookahead(case, seed):
    w, h = case["w"], case["h"]
    return {"w": w, "h": h, "src": _base_picture(_generator(seed), w, h).to(torch.uint8),
            "low": torch.zeros((h // 2, w // 2), dtype=torch.uint8, device="cuda"),
            "mad": [torch.zeros(k, dtype=torch.int32, device="cuda") for k in _maps(w, h)]}


def _prepare_percall(case, seed):
    part = case["part"]
    w, h = xg.PU_W[part], xg.PU_H[part]
    r = np.random.default_rng(seed)
    src = r.integers(16, 236, (64, 64), dtype=np.uint8)
    pred = np.clip(src + np.round(r.laplace(0, 12, src.shape)), 0, 255).astype(np.uint8)
    return {"part": part, "qp": case["qp"], "w": w, "h": h, "src": src, "pred": pred, "rec": np.zeros((64, 64), np.uint8),
            "res": np.zeros(w * h, np.int16), "level": np.zeros(w * h, np.int16), "coef": np.zeros(w * h, np.int16),
            "rres": np.zeros(w * h, np.int16)}


# ---- run ------------------------------------------------------------------------
def run(state):
    return globals()["_run_" + state["kind"]](state)


def _run_me(s):
    sess = s["sess"]
    for i, p in enumerate(s["pics"]):
        sess.set_picture(i - 1, p)
    sess.run(s["prm"])
    sess.results(s["out_np"])
    return s["out"]


def _run_chain(s):
    lib, cur = xg.load(), s["cur"]
    _check(lib.xavs2gpu_copy_h2d(ctypes.c_void_p(s["chain"].source(0)), xg.ptr(cur), cur.nbytes), "copy_h2d")
    s["chain"].launch()
    s["sess"].sync()
    rec = s["recon_np"]
    _check(lib.xavs2gpu_copy_d2h(xg.ptr(rec), ctypes.c_void_p(s["recon_dev"]), rec.nbytes), "copy_d2h")
    return {"recon": s["recon"], **s["views"]}


def _run_serve(s):
    srv = s["srv"]
    for k in range(4):
        for sid, pics in s["streams"]:
            _check(srv.submit(sid, pics[k], tag=k), "submit")
    r = _collect(srv, 4 * len(s["streams"]))
    return r["hash"][np.lexsort((r["frame"], r["stream"]))].view(np.int64)


def _run_tq(s):
    _check(xg.fn("xavs2gpu_tq_batch")(_P(s["blocks"]), s["n"], _P(s["res"]), _P(s["levels"]), _P(s["recon"]),
                                      _P(s["nnz"]), _stream()), "tq_batch")
    return {"levels": s["levels"], "recon": s["recon"], "nnz": s["nnz"]}


def _run_intra(s):
    lib = xg.load()
    _check(lib.xavs2gpu_intra_fill_edges(_P(s["jobs"]), s["n"], _P(s["recon"]), s["w"], s["w"], s["h"],
                                         _P(s["edges"]), s["esize"], _stream()), "intra_fill_edges")
    _check(lib.xavs2gpu_intra_rmd_batch(_P(s["blocks"]), s["n"], _P(s["edges"]), _P(s["src"]), s["w"],
                                        ctypes.byref(s["prm"]), _P(s["out"]), _stream()), "intra_rmd_batch")
    rec = s["out"].view(s["n"], -1)                  # xavs2gpu_intra_result_t: 42 costs, 9 modes, their number
    return {"costs": rec.view(torch.float64)[:, :42], "modes": rec.view(torch.int32)[:, 84:94], "edges": s["edges"]}


def _run_skip(s):
    _check(xg.load().xavs2gpu_skip_costs(ctypes.c_void_p(s["sess"].h), _P(s["cands"]), s["n"], math.sqrt(_lambda_rd()),
                                         s["n_cu"], _P(s["dist"]), _P(s["cost"]), _P(s["best"]), None), "skip_costs")
    return {"dist": s["dist"], "cost": s["cost"], "best": s["best"]}


def _run_loopfilter(s):
    src, dst, w = s["src"], s["dst"], s["w"]
    _check(xg.load().xavs2gpu_loopfilter_picture(_P(src[0]), _P(src[1]), _P(src[2]), _P(dst[0]), _P(dst[1]), _P(dst[2]),
                                                 w, w // 2, w, s["h"], s["level"], _P(s["scus"]), _P(s["lcus"]),
                                                 _stream()), "loopfilter_picture")
    return dst


def _run_lookahead(s):
    _check(xg.load().xavs2gpu_lookahead_picture(_P(s["src"]), s["w"], s["w"], s["h"], _P(s["low"]), s["w"] // 2,
                                                _P(s["mad"][0]), _P(s["mad"][1]), _P(s["mad"][2]), _stream()),
           "lookahead_picture")
    return [s["low"], *s["mad"]]


def _run_percall(s):
    """One block as an encoder's residual coding calls the table: cost of the prediction, residual, transform,
    quantiser and back, reconstruction, its distortion."""
    part, w, p = s["part"], s["w"], xg.ptr
    src, pred, res, level, coef = s["src"], s["pred"], s["res"], s["level"], s["coef"]
    cost = xg.pixel_fn("satd", part)(p(src), 64, p(pred), 64)
    xg.pixel_fn("sub_ps", part)(p(res), w, p(src), p(pred), 64, 64)
    xg.dct_fn("dct", part)(p(res), p(level), w)
    big = max(w, s["h"]) == 64
    n = w * s["h"] // (4 if big else 1)
    # quantiser of an inter TU whose side logs average 4: a step of 2 ** (qp / 8)
    qp = s["qp"]
    nnz = xg.fn("xavs2gpu_quant")(p(level), n, round(32768 * 2 ** (-qp / 8)), 18, (1 << 18) * 5 // 31)
    coef[:] = level
    xg.fn("xavs2gpu_dequant")(p(coef), n, round(2 ** (15 - qp // 8 + qp / 8)), 12 - qp // 8)
    xg.dct_fn("idct", part)(p(coef), p(s["rres"]), w)
    xg.pixel_fn("add_ps", part)(p(s["rec"]), 64, p(pred), p(s["rres"]), 64, w)
    ssd = xg.pixel_fn("ssd", part)(p(src), 64, p(s["rec"]), 64)
    return {"cost": cost, "nnz": nnz, "ssd": ssd, "residual": res, "levels": level[:n], "recon": s["rec"]}


# ---- work -----------------------------------------------------------------------
def work(case):
    """Bytes: each input read and each output written once.  flops: whole-number operations of the path (an absolute
    difference and its accumulation count two, a multiply-add two)."""
    kind = case["kind"]
    w, h = case.get("w", 0), case.get("h", 0)
    px = w * h
    if kind == "me":
        refs, R = case["refs"], case["range"]
        pus = _quadtree(w, h, refs) if case["layout"] == "quadtree" else _leaves(w, h, refs, 5)[0]
        area = int((np.asarray(xg.PU_W)[pus["part"]] * np.asarray(xg.PU_H)[pus["part"]]).sum())
        # PUs with one centre share the differences of their pixels, others each need their own
        shared = case["predictors"] == "zero" and R % 2 == 0
        search = 2 * (px * refs if shared else area) * (2 * R) ** 2
        return {"bytes": px * (1 + refs) + 20 * len(pus), "flops": search + 2 * 17 * area}
    if kind == "chain":
        refs, R = case["refs"], case["range"]
        # about 13 candidates' worth of residual, levels and reconstruction per pixel leave the chain
        return {"bytes": px * (2 + refs) + 4 * 13 * px, "flops": 2 * px * refs * (2 * R) ** 2 + 2 * 17 * 7 * px * refs}
    if kind == "serve":
        n = [case[k] for k in ("n360", "n720", "n1080", "n2160")]
        total = 4 * sum(k * a * b for k, (a, b) in zip(n, SERVE_SIZES))
        return {"bytes": 3 * total, "flops": 2 * total * 2 * ((2 * case["range"]) ** 2 + 17 * 7)}
    if kind == "tq":
        parts = _TQ_PARTS[case["parts"]]
        area = [xg.PU_W[p] * xg.PU_H[p] for p in parts]
        big = [max(xg.PU_W[p], xg.PU_H[p]) == 64 for p in parts]
        mean = sum(4 * a + 2 * (a // 4 if b else a) + 36 for a, b in zip(area, big)) / len(parts)
        mul = sum(2 * 2 * a * (xg.PU_W[p] + xg.PU_H[p]) / (2 if not b else 8) for a, b, p in zip(area, big, parts)) / len(parts)
        return {"bytes": case["n"] * mean, "flops": case["n"] * mul}
    if kind == "intra":
        n = len(synth.intra_level_blocks(w, h))
        return {"bytes": 2 * px + n * (24 + 40 + 376), "flops": 33 * 9 * px * 11}
    if kind == "skip":
        n = sum((w >> lv) * (h >> lv) for lv in (3, 4, 5, 6)) * case["per_cu"]
        return {"bytes": px * (1 + case["refs"]) + n * 68, "flops": 4 * px * case["per_cu"] * 10}
    if kind == "loopfilter":
        return {"bytes": 3 * px + px // 64 * 16, "flops": 30 * px}
    if kind == "lookahead":
        return {"bytes": px + px // 4 + 4 * sum(_maps(w, h)), "flops": 8 * px}
    a = xg.PU_W[case["part"]] * xg.PU_H[case["part"]]
    return {"bytes": 16 * a, "flops": 4 * 16 * a}


# ---- exact ----------------------------------------------------------------------
def exact(case, seed):
    """Whole numbers are compared bit for bit; the doubles of `skip` follow from whole numbers, worked out here from
    the definition: the 8-point Hadamard cost of the prediction plus lambda times the bits."""
    return _exact_skip(case, seed) if case["kind"] == "skip" else None


def _planes(pic):
    """The 16 quarter-pel planes of a picture with their margin of 80, plane 4 * fy + fx: the filters at every position
    up to 4 outside the picture (whose edge samples repeat), the samples further out those nearest to them."""
    pic = pic.double()
    h, w = pic.shape

    def taken(x, axis, lo, n):
        return x.index_select(axis, torch.arange(lo, lo + n, device=x.device).clamp(0, x.shape[axis] - 1))

    def taps(x, f, axis, n):
        return sum(float(t) * x.narrow(axis, k, n) for k, t in enumerate(_TAPS[f]))

    out = []
    for k in range(16):
        fx, fy = k & 3, k >> 2
        if not k:
            out.append(taken(taken(pic, 0, -80, h + 160), 1, -80, w + 160))
            continue
        v = taps(taken(pic, 1, -7, w + 15), fx, 1, w + 8) if fx else taken(pic, 1, -4, w + 8)
        v = taps(taken(v, 0, -7, h + 15), fy, 0, h + 8) if fy else taken(v, 0, -4, h + 8)
        v = torch.floor((v + 2048) / 4096) if fx and fy else torch.floor((v + 32) / 64)
        out.append(taken(taken(v.clamp(0, 255), 0, -76, h + 160), 1, -76, w + 160))
    return torch.stack(out)


def _exact_skip(case, seed):
    w, h, refs, per = case["w"], case["h"], case["refs"], case["per_cu"]
    if w * h * per > 5 * 1920 * 1088:
        return None
    pics, _ = _sequence(seed, refs + 1, w, h, 2, 4, pan=3)
    pics = pics[::-1]
    c, n_cu = _skip_candidates(np.random.default_rng(seed), w, h, refs, per)
    dev = pics[0].device
    cur = pics[0].double()
    flat = torch.cat([_planes(p).reshape(-1) for p in pics[1:]])
    ph, pw = h + 160, w + 160
    hd = torch.ones((1, 1), dtype=torch.float64, device=dev)
    for _ in range(3):
        hd = torch.cat([torch.cat([hd, hd], 1), torch.cat([hd, -hd], 1)], 0)
    dist = np.zeros(len(c), np.float64)
    for lv in (3, 4, 5, 6):
        s = 1 << lv
        sel = np.nonzero(c["size_log2"] == lv)[0]
        grid = torch.arange(s, device=dev)
        quad = ((grid >= s // 2).long()[:, None] * 2 + (grid >= s // 2).long()[None, :])
        for at in range(0, len(sel), max(1, (1 << 24) // (s * s))):
            i = sel[at:at + max(1, (1 << 24) // (s * s))]
            pu = torch.where(torch.from_numpy(c["n_pu"][i] == 4).to(dev)[:, None, None], quad[None], torch.zeros_like(quad)[None])
            y = torch.from_numpy(c["y"][i].astype(np.int64)).to(dev)[:, None, None] + grid[None, :, None]
            x = torch.from_numpy(c["x"][i].astype(np.int64)).to(dev)[:, None, None] + grid[None, None, :]
            pred = []
            for lst in (0, 1):
                ref = torch.from_numpy(c["ref"][i][:, :, lst].astype(np.int64)).to(dev).gather(1, pu.flatten(1)).view(pu.shape)
                mv = [torch.from_numpy(c["mv"][i][:, :, lst, k].astype(np.int64)).to(dev).gather(1, pu.flatten(1)).view(pu.shape)
                      for k in (0, 1)]
                plane = ref.clamp(min=0) * 16 + (mv[1] & 3) * 4 + (mv[0] & 3)
                yy, xx = (y + (mv[1] >> 2) + 80).clamp(0, ph - 1), (x + (mv[0] >> 2) + 80).clamp(0, pw - 1)
                pred.append((flat[(plane * ph + yy) * pw + xx], ref))
            p = torch.where(pred[1][1] >= 0, torch.floor((pred[0][0] + pred[1][0] + 1) / 2), pred[0][0])
            d = (cur[y, x] - p).view(len(i), s // 8, 8, s // 8, 8).permute(0, 1, 3, 2, 4)
            t = (hd @ d @ hd).abs().sum((-1, -2))
            if s == 8:
                cost = torch.floor((t[:, 0, 0] + 2) / 4)
            else:
                t = t.view(len(i), s // 16, 2, s // 16, 2).sum((2, 4))
                cost = torch.floor((t + 2) / 4).sum((1, 2))
            dist[i] = cost.cpu().numpy()
    c = c.reshape(n_cu, per)
    value = dist.reshape(n_cu, per) + math.sqrt(_lambda_rd()) * c["rate"]
    for j in range(1, per):                            # the same motion as an earlier candidate: the largest cost
        for k in range(j):
            same = (c["n_pu"][:, j] == c["n_pu"][:, k]) & (c["ref"][:, j] == c["ref"][:, k]).all((1, 2)) & \
                   (c["mv"][:, j] == c["mv"][:, k]).all((1, 2, 3))
            value[same, j] = 2.0 ** 50
    return {"dist": None, "cost": value.reshape(-1), "best": None}
