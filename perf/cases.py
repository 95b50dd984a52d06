"""The encoder's work as measured cases: whole AVIF encodes, the batched searches that an encoder's
host drives through the device entries of the C ABI, and the frame filters.

A case is a dict of plain values; ``prepare`` makes what a program holds before the call (host
images for the encoder, device buffers for the searches and filters), ``run`` is one pass through the
public entry points.  Every output is a record, a level, a sample or a byte of a file, all of them
exact by contract (the f32 fields of the records too: their summation order is fixed), so the records
are returned as bytes.
"""
import ctypes as C
import math

import numpy as np
import torch

import maroontree_b200 as mt
from maroontree_b200 import abi
from maroontree_b200 import encoder as enc

ALL_MODES = tuple(range(13))
# The transform types that each level tries for every mode.
LEVEL_TYPES = {4: (abi.TX_DCT_DCT, abi.TX_ADST_ADST, abi.TX_IDTX, abi.TX_ADST_DCT, abi.TX_DCT_ADST),
               8: abi.TX_2D_SCAN_TYPES, 16: (abi.TX_DCT_DCT, abi.TX_ADST_ADST, abi.TX_IDTX)}


def listed():
    return [
        # Encodes of host RGB to AVIF bytes.  A thumbnail with ragged sides: latency of one call.
        dict(name="encode_thumb_420", kind="encode", w=150, h=101, chroma=420, quality=50),
        # A small full-chroma picture (icons, avatars, product shots).
        dict(name="encode_512_444", kind="encode", w=512, h=512, chroma=444, quality=60),
        # The ordinary photo: 1080p at 4:2:0.
        dict(name="encode_1080p_420", kind="encode", w=1920, h=1080, chroma=420, quality=60),
        # The largest frame the benchmark names, two tiles.
        dict(name="encode_4096_444", kind="encode", w=4096, h=4096, chroma=444, quality=60),
        # A service's queue: uneven sizes and qualities, both chroma formats, in one call.
        dict(name="encode_batch_uneven", kind="batch", count=12, lo=64, hi=2048, pick=11),
        # One 8x8 level of the partition search over a frame: every block, mode and 2-D type.
        dict(name="level8_1080p", kind="level", n=8, w=1920, h=1080, quality=60, deltas=False),
        # The leaf searches' mode loops over a frame, by leaf size.
        dict(name="leaf16_modes_1080p", kind="leaf", n=16, refine=False, w=1920, h=1080, quality=60, wsse=False),
        dict(name="leaf32_modes_1080p", kind="leaf", n=32, refine=False, w=1920, h=1080, quality=60, wsse=False),
        dict(name="leaf64_quads_1080p", kind="leaf64", grid=False, w=1920, h=1080, quality=60),
        # The leaves' chroma searches with the winners' levels and samples: 4:2:0 and 4:4:4.
        dict(name="uv16_420_1080p", kind="uv", leaf=16, chroma=420, w=1920, h=1080, quality=60),
        dict(name="uv32_444_1080p", kind="uv", leaf=32, chroma=444, w=1920, h=1080, quality=60),
        # Deblocking and CDEF of a whole decided frame.
        dict(name="filters_4096_444", kind="filters", w=4096, h=4096, chroma=444, quality=60),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["encode", "encode", "batch", "level", "leaf", "leaf", "leaf64", "uv", "uv", "filters"])
    quality = rng.randint(30, 90)
    chroma = rng.choice([420, 444])
    if kind == "encode":
        return dict(kind=kind, w=_log(rng, 64, 2048), h=_log(rng, 64, 2048), chroma=chroma, quality=quality)
    if kind == "batch":
        return dict(kind=kind, count=rng.randint(2, 12), lo=64, hi=_log(rng, 256, 2048), pick=rng.randint(0, 1 << 20))
    if kind == "filters":
        return dict(kind=kind, w=_log(rng, 64, 4096), h=_log(rng, 64, 4096), chroma=chroma, quality=quality)
    size = dict(w=_log(rng, 128, 1920), h=_log(rng, 128, 1080), quality=quality)
    if kind == "level":
        return dict(kind=kind, n=rng.choice([4, 8, 16]), deltas=rng.random() < 0.3, **size)
    if kind == "leaf":
        n = rng.choice([8, 16, 32])
        return dict(kind=kind, n=n, refine=n != 32 and rng.random() < 0.4, wsse=rng.random() < 0.5, **size)
    if kind == "leaf64":
        return dict(kind=kind, grid=rng.random() < 0.5, **size)
    return dict(kind=kind, leaf=rng.choice([16, 32]), chroma=chroma, **size)


# ---- inputs ----

def _rng(seed, salt=0):
    return np.random.default_rng((int(seed) * 1000003 + salt) & 0x7FFFFFFF)


def _image(w, h, seed, noise=4.0):
    """A (3, h, w) float image on the GPU like the benchmark's generator: sinusoids, hard-edged
    rectangles (half of them rotated), a texture band, a gradient quadrant, and noise."""
    r = _rng(seed)
    y = torch.arange(h, device="cuda", dtype=torch.float32)[:, None]
    x = torch.arange(w, device="cuda", dtype=torch.float32)[None, :]
    img = torch.full((3, h, w), 128.0, device="cuda")
    for _ in range(6):
        f, th = r.uniform(1, 40), r.uniform(0, math.pi)
        arg = 2 * math.pi * f * (math.cos(th) * x / w + math.sin(th) * y / h)
        for c in range(3):
            img[c] += r.uniform(0, 60) * torch.sin(arg + r.uniform(0, 2 * math.pi))
    for k in range(12):
        cx, cy = r.uniform(0, w), r.uniform(0, h)
        sw, sh = r.uniform(w / 32, w / 4), r.uniform(w / 32, w / 4)
        a = r.uniform(0, math.pi) if k >= 6 else 0.0
        u = (x - cx) * math.cos(a) + (y - cy) * math.sin(a)
        v = (y - cy) * math.cos(a) - (x - cx) * math.sin(a)
        inside = (u.abs() <= sw / 2) & (v.abs() <= sh / 2)
        for c in range(3):
            img[c].masked_fill_(inside, float(r.integers(0, 256)))
    b0, b1 = h // 4, h // 4 + max(1, h // 8)
    img[:, b0:b1] += 40 * torch.sin(2 * math.pi * x / 64) * torch.sin(2 * math.pi * y[b0:b1] / 64)
    img[:, h // 2:, w // 2:] = 255.0 * ((x[:, w // 2:] - w // 2) + (y[h // 2:] - h // 2)) / (w / 2 + h / 2)
    g = torch.Generator(device="cuda").manual_seed(int(seed) + 17)
    img += noise * torch.randn(img.shape, generator=g, device="cuda")
    return img.round_().clamp_(0, 255)


def _host_rgb(w, h, seed):
    return np.ascontiguousarray(_image(w, h, seed).to(torch.uint8).permute(1, 2, 0).contiguous().cpu().numpy())


def _pad8(p):
    h, w = p.shape
    return torch.nn.functional.pad(p[None, None], (0, -w % 8, 0, -h % 8), mode="replicate")[0, 0]


def _planes(w, h, chroma, seed):
    """Padded source planes Y, U, V (float, 8-bit values) of a textured image: U and V the blue and red
    channels, averaged over 2x2 cells at 4:2:0."""
    img = _image(w, h, seed)
    y = _pad8((0.299 * img[0] + 0.587 * img[1] + 0.114 * img[2]).round())
    uv = [_pad8(img[2]), _pad8(img[0])]
    if chroma == 420:
        uv = [torch.nn.functional.avg_pool2d(p[None, None], 2)[0, 0].round() for p in uv]
    return [y] + uv


def _u16(p):
    return p.to(torch.int16).contiguous()


def _coded(p, seed, amp=3):
    """A reconstruction of the plane: the source with a small coding error."""
    g = torch.Generator(device="cuda").manual_seed(int(seed) + 29)
    return (p + torch.randint(-amp, amp + 1, p.shape, generator=g, device="cuda")).clamp(0, 255)


def _bytes(a):
    return torch.from_numpy(np.frombuffer(np.ascontiguousarray(a).tobytes(), np.uint8).copy()).cuda()


def _empty(n):
    return torch.zeros(max(int(n), 1), dtype=torch.uint8, device="cuda")


def _grid(w8, h8, n, r):
    """Every n x n block of the padded frame in raster order: positions and flags (the neighbour
    availability of a z-order walk; a random filter type)."""
    ys, xs = np.meshgrid(np.arange(0, h8 - n + 1, n), np.arange(0, w8 - n + 1, n), indexing="ij")
    px, py = xs.ravel(), ys.ravel()
    bx, by = px // n, py // n
    tr = (py > 0) & (px + n < w8) & ((bx % 2 == 0) | (by % 2 == 0))
    bl = (px > 0) & (py + n < h8) & (bx % 2 == 1) & (by % 2 == 0)
    ft = r.random(len(px)) < 0.5
    return px, py, tr * abi.CAND_HAVE_TR + bl * abi.CAND_HAVE_BL + ft * abi.CAND_FILTER_TYPE


def _ctx(r, shape):
    """Neighbouring blocks' coefficient result contexts."""
    b = r.integers(1, 64, size=shape) | r.choice(np.array([0x00, 0x40, 0x80]), size=shape)
    return np.where(r.random(shape) < 0.3, 0x40, b).astype(np.uint8)


def _mode_major(dtype, px, py, flags, modes, deltas=(0,)):
    """One job per (mode, delta, block), blocks innermost."""
    md = [(m, d) for m in modes for d in (deltas if abi.V_PRED <= m <= abi.D67_PRED else (0,))]
    jobs = np.zeros(len(md) * len(px), dtype)
    jobs["px"], jobs["py"], jobs["flags"] = np.tile(px, len(md)), np.tile(py, len(md)), np.tile(flags, len(md))
    jobs["mode"] = np.repeat([m for m, _ in md], len(px))
    jobs["angle_delta"] = np.repeat([d for _, d in md], len(px))
    return jobs


def _laws(quality, chroma, plane, n):
    """The frame's quantiser, QM row, lambdas and default costs for n x n blocks of a plane."""
    sub = 2 if chroma == 420 else 0
    qidx = mt.quality_to_q(quality)
    levels = mt.qm_levels(qidx, sub)
    level = levels[1 if plane else 0]
    q = mt.quant_new_chroma(qidx, 0, 0, 8, level) if plane else mt.quant_new(qidx, 8, level)
    lam = mt.rd_lambdas(qidx, mt.quant_new(qidx, 8, levels[0]).dc_q, sub)
    qm = mt.qm_row(level, 1 if plane else 0, n) if level < 15 else None
    costs = mt.coef_costs(mt.coef_cdfs_default(mt.qcat(qidx), n, n, 1 if plane else 0))
    return q, lam, None if qm is None else _bytes(qm), _bytes(np.frombuffer(bytes(costs), np.uint8))


def _sizes(case):
    r = _rng(case["pick"], 5)
    lo, hi = math.log(case["lo"]), math.log(case["hi"])
    return [(int(round(math.exp(r.uniform(lo, hi)))), int(round(math.exp(r.uniform(lo, hi)))),
             int(r.integers(30, 91)), int(r.choice([420, 444]))) for _ in range(case["count"])]


# ---- one prepare and run per kind ----

def _config(quality, chroma):
    return enc.config(quality=quality, chroma=0 if chroma == 420 else 2)


class _File:
    """Where a program keeps the encoded file: a buffer of a byte a sample, the bytes past the file's end zero."""

    def __init__(self, w, h, chroma):
        self.buf, self.n = np.zeros(w * h * (6 if chroma == 444 else 3) // 2 + 4096, np.uint8), 0

    def put(self, data):
        n = len(data)
        self.buf[:n] = np.frombuffer(data, np.uint8)
        self.buf[n:self.n] = 0
        self.n = n
        return dict(length=n, file=self.buf)


def _prepare_encode(case, seed):
    w, h, chroma = case["w"], case["h"], case["chroma"]
    return dict(rgb=_host_rgb(w, h, seed), cfg=_config(case["quality"], chroma), file=_File(w, h, chroma))


def _run_encode(s):
    return s["file"].put(enc.encode_rgb8(s["rgb"], s["cfg"]))


def _prepare_batch(case, seed):
    sizes = _sizes(case)
    return dict(imgs=[_host_rgb(w, h, seed * 64 + i) for i, (w, h, _, _) in enumerate(sizes)],
                cfgs=[_config(q, ch) for _, _, q, ch in sizes], files=[_File(w, h, ch) for w, h, _, ch in sizes])


def _run_batch(s):
    return [f.put(data) for f, data in zip(s["files"], enc.encode_rgb8_batch(s["imgs"], s["cfgs"]))]


def _luma(case, seed):
    p = _planes(case["w"], case["h"], 444, seed)[0]
    return _u16(p), _u16(_coded(p, seed)), p.shape[1], p.shape[0]


def _prepare_level(case, seed):
    n = case["n"]
    src, rec, w8, h8 = _luma(case, seed)
    q, lam, qm, costs = _laws(case["quality"], 420, 0, n)
    r = _rng(seed, 1)
    px, py, flags = _grid(w8, h8, n, r)
    blocks = np.zeros(len(px), abi.BLOCK8_DTYPE)
    blocks["px"], blocks["py"], blocks["flags"] = px, py, flags
    blocks["dcs_ctx"] = r.integers(0, 3, size=len(px))
    blocks["mode_bits"] = r.uniform(1, 7, (len(px), 13))
    rows = []
    for m in ALL_MODES:
        for d in ((-3, 0, 3) if case["deltas"] and abi.V_PRED <= m <= abi.D67_PRED else (0,)):
            for t in LEVEL_TYPES[n]:
                rows.append((m, d, t, abi.COMBO_NO_TRELLIS if n == 4 and t == abi.TX_IDTX else 0, 1.5 if d else 0.0))
    combos = np.array(rows, abi.COMBO_DTYPE)
    nb, nc = len(blocks), len(combos)
    prm = mt.chain_params(w8, h8, tx_size=n, trellis_lambda0=lam.trellis_lambda0, mode_lambda=lam.mode_lambda,
                          satd_scale=lam.satd_scale, satd_bridge=lam.satd_bridge, vis=(case["w"], case["h"]))
    lib = mt.load()
    scratch = _empty(getattr(lib, f"mt_rdo_level{n}_scratch_bytes")(nb, nc))
    return dict(entry=getattr(lib, f"mt_rdo_level{n}_device"), src=src, rec=rec, prm=prm, q=q, qm=qm, costs=costs,
                blocks=_bytes(blocks), combos=_bytes(combos), nb=nb, nc=nc, scratch=scratch,
                best=_empty(nb * abi.BEST_DTYPE.itemsize), results=_empty(nb * nc * abi.RESULT_DTYPE.itemsize))


def _stream():
    return torch.cuda.current_stream().cuda_stream


def _ok(rc, what):
    if rc != abi.MT_OK:
        raise mt.MtError(rc, what)


def _p(t):
    return None if t is None else t.data_ptr()


def _run_level(s):
    _ok(s["entry"](_p(s["src"]), _p(s["rec"]), C.byref(s["prm"]), C.byref(s["q"]), _p(s["qm"]), _p(s["costs"]),
                   _p(s["blocks"]), s["nb"], _p(s["combos"]), s["nc"], _p(s["best"]), _p(s["results"]),
                   _p(s["scratch"]), _stream()), "mt_rdo_level_device")
    return dict(best=s["best"], results=s["results"])


def _prepare_leaf(case, seed):
    n, refine = case["n"], case["refine"]
    src, rec, w8, h8 = _luma(case, seed)
    q, lam, qm, costs = _laws(case["quality"], 444 if refine else 420, 0, n)
    r = _rng(seed, 2)
    px, py, flags = _grid(w8, h8, n, r)
    jobs = _mode_major(abi.LEAF8_JOB_DTYPE, px, py, flags, (abi.DC_PRED,) if refine else ALL_MODES)
    if refine:  # one winner per block
        jobs["mode"] = r.integers(0, 13, size=len(jobs))
    jobs["dcs_ctx"] = np.resize(r.integers(0, 3, size=len(px)), len(jobs))
    jobs["syntax_bits"] = r.uniform(1, 7, size=len(jobs))
    prm = mt.split16_params(w8, h8, trellis_lambda0=lam.trellis_lambda0, rd_lambda=lam.lambda_d, band_tilt=1.9,
                            wsse_scale=1.0 if case["wsse"] else 0.0, tx_search=refine, tx_guard_shift=5,
                            vis=(case["w"], case["h"]))
    what = f"mt_leaf{n}_tx_refine_device" if refine else f"mt_leaf{n}_luma_device"
    nj = len(jobs)
    out = dict(results=_empty(nj * abi.LEAF8_RESULT_DTYPE.itemsize))
    if refine:  # the winners' levels and samples are what gets coded
        out.update(levels=torch.zeros(nj, n * n, dtype=torch.int32, device="cuda"),
                   samples=torch.zeros(nj, n * n, dtype=torch.int16, device="cuda"))
    return dict(entry=getattr(mt.load(), what), src=src, rec=rec, prm=prm, q=q, qm=qm, costs=costs, jobs=_bytes(jobs),
                n=nj, out=out)


def _run_leaf(s):
    o = s["out"]
    _ok(s["entry"](_p(s["src"]), _p(s["rec"]), C.byref(s["prm"]), C.byref(s["q"]), _p(s["qm"]), _p(s["costs"]),
                   _p(s["jobs"]), s["n"], _p(o["results"]), _p(o.get("levels")), _p(o.get("samples")), _stream()),
        "mt_leaf_device")
    return o


def _prepare_leaf64(case, seed):
    grid = case["grid"]
    n = 16 if grid else 32
    src, rec, w8, h8 = _luma(case, seed)
    q, lam, qm, costs = _laws(case["quality"], 420, 0, n)
    r = _rng(seed, 3)
    px, py, flags = _grid(w8, h8, 64, r)
    jobs = _mode_major(abi.GRID16_JOB_DTYPE if grid else abi.QUAD32_JOB_DTYPE, px, py, flags,
                       (abi.DC_PRED,) if grid else ALL_MODES)
    nj = len(jobs)
    if grid:  # the tx_depth-2 trial of each block's winning mode
        jobs["mode"] = r.integers(0, 13, size=nj)
        jobs["a_coef"], jobs["l_coef"] = _ctx(r, (nj, 16)), _ctx(r, (nj, 16))
        jobs["depth_bits"] = r.uniform(-1, 3, size=nj)
    else:
        jobs["dcs_ctx"] = r.integers(0, 3, size=(nj, 4))
    jobs["mode_bits"], jobs["delta_bits"] = r.uniform(1, 7, size=nj), r.uniform(0.5, 3.5, size=nj)
    prm = mt.split16_params(w8, h8, trellis_lambda0=lam.trellis_lambda0, rd_lambda=lam.lambda_d, band_tilt=1.9,
                            wsse_scale=1.0, vis=(case["w"], case["h"]))
    lib = mt.load()
    out = dict(results=_empty(nj * (abi.GRID16_RESULT_DTYPE if grid else abi.QUAD32_RESULT_DTYPE).itemsize))
    if grid:
        out["levels"] = torch.zeros(nj, 4096, dtype=torch.int32, device="cuda")
    return dict(entry=lib.mt_grid16_luma_device if grid else lib.mt_quad32_luma_device, src=src, rec=rec, prm=prm, q=q,
                qm=qm, costs=costs, jobs=_bytes(jobs), n=nj, out=out)


def _run_leaf64(s):
    o = s["out"]
    args = [_p(s["src"]), _p(s["rec"]), C.byref(s["prm"]), C.byref(s["q"]), _p(s["qm"]), _p(s["costs"]), _p(s["jobs"]),
            s["n"], _p(o["results"])]
    if "levels" in o:
        args.append(_p(o["levels"]))
    _ok(s["entry"](*args, _stream()), "mt_leaf64_device")
    return o


def _prepare_uv(case, seed):
    leaf, chroma = case["leaf"], case["chroma"]
    n = leaf // 2 if chroma == 420 else leaf
    y, u, v = _planes(case["w"], case["h"], chroma, seed)
    q, lam, qm, costs = _laws(case["quality"], chroma, 1, n)
    r = _rng(seed, 4)
    px, py, flags = _grid(y.shape[1], y.shape[0], leaf, r)
    dtype = {8: abi.UV16_JOB_DTYPE, 16: abi.UV16_444_JOB_DTYPE, 32: abi.UV32_444_JOB_DTYPE}[n]
    jobs = np.zeros(len(px), dtype)
    jobs["px"], jobs["py"], jobs["flags"] = px, py, flags
    jobs["y_mode"] = r.integers(0, 13, size=len(px))
    jobs["a_coef"], jobs["l_coef"] = _ctx(r, jobs["a_coef"].shape), _ctx(r, jobs["l_coef"].shape)
    s = 1 if chroma == 420 else 0
    prm = mt.split16_params(u.shape[1], u.shape[0], trellis_lambda0=lam.trellis_lambda0, rd_lambda=lam.mode_lambda,
                            wsse_scale=1.0, vis=((case["w"] + s) >> s, (case["h"] + s) >> s))
    uvp = mt.uv16_params(y.shape[1], joint_k=4, angle_deltas=True, dir_lambda=lam.lambda_d)
    mode_costs = mt.uv_mode_costs(mt.uv_mode_cdfs_default())
    nj = len(jobs)
    return dict(entry=getattr(mt.load(), f"mt_pick_uv{leaf}_{chroma}_device"), prm=prm, uvp=uvp, q=q, qm=qm,
                planes=[_u16(u), _u16(v), _u16(_coded(u, seed + 1)), _u16(_coded(v, seed + 2)), _u16(_coded(y, seed))],
                costs=costs, mode_costs=_bytes(np.frombuffer(bytes(mode_costs), np.uint8)), jobs=_bytes(jobs), n=nj,
                out=dict(results=_empty(nj * abi.UV16_RESULT_DTYPE.itemsize),
                         levels=torch.zeros(nj, 2 * n * n, dtype=torch.int32, device="cuda"),
                         samples=torch.zeros(nj, 2 * n * n, dtype=torch.int16, device="cuda")))


def _run_uv(s):
    o = s["out"]
    _ok(s["entry"](*[_p(t) for t in s["planes"]], C.byref(s["prm"]), C.byref(s["uvp"]), C.byref(s["q"]), _p(s["qm"]),
                   _p(s["costs"]), _p(s["mode_costs"]), _p(s["jobs"]), s["n"], _p(o["results"]), _p(o["levels"]),
                   _p(o["samples"]), _stream()), "mt_pick_uv_device")
    return o


def _prepare_filters(case, seed):
    sub = 1 if case["chroma"] == 420 else 0
    qidx = mt.quality_to_q(case["quality"])
    src = _planes(case["w"], case["h"], case["chroma"], seed)
    h8, w8 = src[0].shape
    r = _rng(seed, 6)
    # block sizes: each 64x64 superblock split evenly into 8x8 .. 64x64 blocks, mostly small ones
    side = r.choice(np.array([2, 2, 2, 4, 4, 8, 16]), size=(-(-h8 // 64), -(-w8 // 64)))
    side = np.repeat(np.repeat(side, 16, 0), 16, 1)[:h8 // 4, :w8 // 4].astype(np.uint8)
    ys, xs = np.mgrid[0:h8 // 4, 0:w8 // 4]
    maps = [side, side, (xs % side == 0).astype(np.uint8), (ys % side == 0).astype(np.uint8), side, side]
    rec = []
    for k, p in enumerate(src):  # coding error: a step per 8x8 block and noise, both by superblock
        s = sub if k else 0
        amp = torch.from_numpy(r.choice([0.5, 1.0, 2.0, 4.0, 7.0], size=(-(-h8 // 64), -(-w8 // 64)))).float().cuda()
        big = 64 >> s
        amp = amp.repeat_interleave(big, 0).repeat_interleave(big, 1)[:p.shape[0], :p.shape[1]]
        step = torch.from_numpy(r.uniform(-1, 1, size=(h8 // 8, w8 // 8))).float().cuda()
        step = step.repeat_interleave(8 >> s, 0).repeat_interleave(8 >> s, 1)
        g = torch.Generator(device="cuda").manual_seed(seed + 31 + k)
        noise = torch.rand(p.shape, generator=g, device="cuda") * 2 - 1
        rec.append(_u16((p + amp * (step + noise)).round().clamp(0, 255)))
    prm = abi.DeblockFrameParams()
    prm.w8, prm.h8, prm.disp_w, prm.disp_h = w8, h8, case["w"], case["h"]
    prm.sub_x, prm.sub_y, prm.mono, prm.bd = sub, sub, 0, 8
    cdef = mt.cdef_params(case["w"], case["h"], sub, sub, qidx)
    lib = mt.load()
    units = (-(-w8 // 64)) * (-(-h8 // 64))
    return dict(src=[_u16(p) for p in src], rec=rec, out=[torch.zeros_like(p) for p in rec],
                maps=[torch.from_numpy(np.ascontiguousarray(m)).cuda() for m in maps],
                skip=_bytes((r.random((h8 // 8, w8 // 8)) < 0.3).astype(np.uint8)), prm=prm, cdef=cdef,
                levels=mt.loop_filter_levels(qidx, sub, sub), grid=np.zeros(units, np.uint8),
                scratch=_empty(lib.mt_deblock_frame_scratch_bytes(C.byref(prm))),
                cdef_scratch=_empty(lib.mt_cdef_scratch_bytes(C.byref(cdef))))


def _run_filters(s):
    lib = mt.load()
    ly, luv, _ = s["levels"]
    decision = abi.CdefDecision()
    _ok(lib.mt_deblock_frame_device_to(*[_p(t) for t in s["rec"]], *[_p(t) for t in s["out"]],
                                       *[_p(t) for t in s["maps"]], C.byref(s["prm"]), ly, luv, luv, _p(s["scratch"]),
                                       _stream()), "mt_deblock_frame_device_to")
    _ok(lib.mt_cdef_frame_device(*[_p(t) for t in s["out"]], *[_p(t) for t in s["src"]], _p(s["skip"]),
                                 C.byref(s["cdef"]), _p(s["cdef_scratch"]), C.byref(decision),
                                 s["grid"].ctypes.data, _stream()), "mt_cdef_frame_device")
    return dict(planes=s["out"], grid=s["grid"], decision=np.frombuffer(bytes(decision), np.uint8))


_KINDS = {"encode": (_prepare_encode, _run_encode), "batch": (_prepare_batch, _run_batch),
          "level": (_prepare_level, _run_level), "leaf": (_prepare_leaf, _run_leaf),
          "leaf64": (_prepare_leaf64, _run_leaf64), "uv": (_prepare_uv, _run_uv),
          "filters": (_prepare_filters, _run_filters)}


def prepare(case, seed):
    state = _KINDS[case["kind"]][0](case, seed)
    state["kind"] = case["kind"]
    return state


def run(state):
    return _KINDS[state["kind"]][1](state)


# ---- the work of a pass ----

# Integer and f32 operations of one n x n candidate chain per sample: residual, quantisation with the
# QM, dequantisation, trellis and rate (about 90), and two n-point passes each way.
def _chain_ops(n):
    return 90 + 4 * 4 * math.log2(n)


def work(case):
    kind = case["kind"]
    if kind == "batch":
        parts = [work(dict(kind="encode", w=w, h=h, chroma=ch, quality=q)) for w, h, q, ch in _sizes(case)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    px = case["w"] * case["h"]
    chroma = 2 if case.get("chroma") == 444 else 0.5
    if kind == "encode":  # RGB in, the file (about a tenth of a byte a sample) out; 91 chains a block and chroma's
        return {"bytes": px * (3 + 0.15 * (1 + chroma)), "flops": px * (91 + chroma) * _chain_ops(8)}
    if kind == "filters":  # recon and source in, planes out; deblocking, 12 CDEF strengths and the chosen one
        samples = px * (1 + chroma)
        return {"bytes": samples * 6, "flops": samples * 13 * 60}
    if kind == "level":
        n = case["n"]
        md = 13 + (16 if case["deltas"] else 0)
        cands = (px / (n * n)) * md * len(LEVEL_TYPES[n])
        return {"bytes": px * 4 + cands * 32, "flops": cands * n * n * _chain_ops(n)}
    if kind == "leaf":
        n = case["n"]
        chains = (7 if n == 8 else 5) if case["refine"] else 13
        out = px * 6 if case["refine"] else (px / (n * n)) * 13 * 36
        return {"bytes": px * 4 + out, "flops": px * chains * _chain_ops(n)}
    if kind == "leaf64":
        chains, n = (1, 16) if case["grid"] else (13, 32)
        return {"bytes": px * 4 + (px * 4 if case["grid"] else 0), "flops": px * chains * _chain_ops(n)}
    # uv: DC, CfL and four priced modes per plane, the ranking's predictions
    n = case["leaf"] // (2 if case["chroma"] == 420 else 1)
    samples = px * chroma
    ranked = 60 if n == 8 else 20
    return {"bytes": samples * (4 + 6) + px * 2, "flops": samples * (6 * _chain_ops(n) + ranked * 16)}


def exact(case, seed):
    """Every output is a whole number or a byte (of a file, or of a record whose fields are fixed to the
    bit), so there is nothing that a computation in 64 bits would be nearer to."""
    return None
