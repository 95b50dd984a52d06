"""The leaf searches that give each block N lanes of a warp, where such a split can go wrong: job counts
around a warp's and a CTA's blocks, rejected jobs among good ones, displayed windows that cut a block at
every remainder of the weighted SSE's tiles, levels of every size class (empty blocks, above 63, Golomb
tails), no trellis, a tight tx-search bound.  Bit for bit against the oracle."""
import os

import numpy as np
import pytest

from maroontree_b200 import abi, synth

W, H = 208, 144


def _case(kind, seed):
    """Source, reconstruction of a content kind."""
    rng = np.random.default_rng(seed)
    if kind == "flat":  # every block predicted exactly somewhere, small residuals elsewhere
        src = np.full((H, W), 90, np.uint16)
        src[:, W // 2:] += rng.integers(0, 3, (H, W - W // 2)).astype(np.uint16)
    elif kind == "hard":  # full-scale noise: long runs of large levels
        src = np.where(rng.random((H, W)) < 0.5, 0, 255).astype(np.uint16)
    else:
        src = synth.rgb_to_luma(synth.generate_rgb(W, H, seed))
    return src, synth.synthetic_recon(src, seed + 5)


def _jobs(family, seed):
    modes, deltas = range(13), (-2, 0, 3)
    if family == "quad32" or family == "grid16":
        return synth.leaf64_jobs(W, H, modes, deltas, seed=seed, grid=family == "grid16")
    return synth.leaf8_jobs(W, H, modes, deltas, seed=seed, n=32 if family == "leaf32" else 16)


@pytest.mark.gpu
@pytest.mark.parametrize("family", ["leaf16", "refine16", "leaf32", "quad32", "grid16"])
@pytest.mark.parametrize("n,kind,qidx,vis,wsse,lam0", [
    (1, "photo", 70, None, 0.0, 0.05),        # one block: idle lanes in its warp
    (2, "hard", 1, (203, 139), 1.0, 0.05),    # the finest steps: Golomb levels
    (7, "flat", 200, (197, 133), 0.5, 0.3),   # empty blocks
    (9, "hard", 40, (190, 100), 1.0, 0.0),    # no trellis; blocks past the displayed frame
    (41, "photo", 1, (201, 130), 0.0, 0.9),
    (83, "photo", 140, (199, 141), 1.0, 0.2),
])
def test_lane_leaves_match_oracle(mt_lib, oracle_lib, cuda, family, n, kind, qidx, vis, wsse, lam0):
    src, rec = _case(kind, qidx + n)
    size = 32 if family in ("leaf32", "quad32") else 16
    qm_level = 15 if qidx == 1 else 4 + qidx % 9
    q = oracle_lib.quant_new(qidx, 8, qm_level)
    qm = oracle_lib.qm_row(qm_level, 0, size) if qm_level < 15 else None
    c = oracle_lib.default_cdfs(oracle_lib.qcat(qidx), size)
    rng = np.random.default_rng(n)
    jobs = _jobs(family, n)
    jobs = jobs[rng.permutation(len(jobs))[:n]]  # mixed modes in a warp
    for i in range(2, n, 5):  # rejected: outside the frame, or no such mode
        if i % 2:
            jobs["mode"][i] = 13
        else:
            jobs["px"][i] = W - 8
    prm = mt_lib.split16_params(W, H, trellis_lambda0=lam0, rd_lambda=0.02 if kind == "hard" else 0.5 * qidx + 1.0,
                                band_tilt=1.9 if n % 2 else 0.0, wsse_scale=wsse, tx_guard_shift=2, vis=vis,
                                skip_bits=[(2.5 + k, 0.4) for k in range(13)] if n % 3 else None)
    costs, threads = mt_lib.coef_costs(c), os.cpu_count() or 1
    args, oargs = (src, rec, prm, q, qm, costs, jobs), (src, rec, prm, q, qm, c, jobs)
    if family == "quad32":
        got, want = [mt_lib.quad32_luma(*args)], [oracle_lib.quad32_luma(*oargs, threads=threads)]
    elif family == "grid16":
        got = mt_lib.grid16_luma(*args, want_cf=True)
        want = oracle_lib.grid16_luma(*oargs, threads=threads, want_cf=True)
    elif family == "leaf32":
        got = mt_lib.leaf32(*args, want_cf=True, want_rec=True)
        want = oracle_lib.leaf32(*oargs, threads=threads)
    else:
        refine = family == "refine16"
        got = mt_lib.leaf16(*args, refine=refine, want_cf=True, want_rec=True)
        want = oracle_lib.leaf16(*oargs, refine=refine, threads=threads)
    for a, b in zip(got, want):
        assert np.asarray(a).tobytes() == np.asarray(b).tobytes()


@pytest.mark.gpu
@pytest.mark.parametrize("over", [-1, 0, 25])
def test_leaf16_cta_sizes_match_oracle(mt_lib, oracle_lib, cuda, over):
    """Job counts around the one from which the 16x16 mode loop runs in CTAs of
    24 jobs (96 per SM), the last CTA full, with one job, or with all but one."""
    import torch

    n = 96 * torch.cuda.get_device_properties(0).multi_processor_count + over
    src, rec = _case("photo", 9)
    q, qm = oracle_lib.quant_new(90, 8, 6), oracle_lib.qm_row(6, 0, 16)
    c = oracle_lib.default_cdfs(oracle_lib.qcat(90), 16)
    jobs = _jobs("leaf16", 9)
    jobs = jobs[np.random.default_rng(n).integers(0, len(jobs), n)]
    jobs["mode"][n - 1:] = 13  # rejected
    prm = mt_lib.split16_params(W, H, trellis_lambda0=0.05, rd_lambda=40.0, band_tilt=1.9, wsse_scale=0.5)
    got = mt_lib.leaf16(src, rec, prm, q, qm, mt_lib.coef_costs(c), jobs, want_cf=True, want_rec=True)
    want = oracle_lib.leaf16(src, rec, prm, q, qm, c, jobs, threads=os.cpu_count() or 1)
    for a, b in zip(got, want):
        assert np.asarray(a).tobytes() == np.asarray(b).tobytes()


@pytest.mark.gpu
@pytest.mark.parametrize("form", ["16_420", "32_420", "16_444", "32_444"])
@pytest.mark.parametrize("kind,qidx,cut,wsse,lam0,joint_k,ad", [
    ("photo", 70, (0, 0), 0.0, 0.05, 1, True),
    ("hard", 1, (5, 3), 1.0, 0.05, 12, True),    # the finest steps; shortlists past one step's candidates
    ("flat", 200, (9, 50), 0.5, 0.3, 5, True),   # empty blocks, leaves past the displayed frame
    ("hard", 40, (17, 6), 1.0, 0.0, 4, False),   # no trellis, no deltas
    ("photo", 130, (2, 1), 1.0, 0.6, 7, True),
])
def test_lane_chroma_matches_oracle(mt_lib, oracle_lib, cuda, form, kind, qidx, cut, wsse, lam0, joint_k, ad):
    leaf, sub = int(form[:2]), form.endswith("420")
    n = leaf // 2 if sub else leaf
    y, yr = _case(kind, qidx)
    (u, ur), (v, vr) = _case(kind, qidx + 1), _case("photo", qidx + 2)
    if sub:
        u, ur, v, vr = [np.ascontiguousarray(a[::2, ::2]) for a in (u, ur, v, vr)]
    qm_level = 15 if qidx == 1 else 3 + qidx % 9
    q = oracle_lib.quant_new_chroma(qidx, 0, 0, 8, qm_level)
    qm = oracle_lib.qm_row(qm_level, 1, n) if qm_level < 15 else None
    ch, cw = u.shape
    prm = mt_lib.split16_params(cw, ch, trellis_lambda0=lam0, rd_lambda=0.03 if kind == "hard" else 0.4 * qidx + 1.0,
                                band_tilt=0.7, wsse_scale=wsse, vis=(cw - cut[0], ch - cut[1]),
                                skip_bits=[(2.0 + 0.3 * k, 0.5) for k in range(13)] if qidx > 100 else None)
    uvp = mt_lib.uv16_params(W, joint_k=joint_k, angle_deltas=ad, dir_lambda=0.3 * qidx + 0.5)
    if form == "16_420":
        jobs = synth.uv16_jobs(W, H, qidx)
    elif form == "32_444":
        jobs = synth.uv32_444_jobs(W, H, qidx)
    else:
        jobs = synth.uv16_444_jobs(W, H, qidx, leaf=leaf)
    jobs["px"][1] = W - leaf + 4  # off the leaf grid: rejected
    jobs["y_mode"][2] = 13
    qctx = oracle_lib.qcat(qidx)
    got = getattr(mt_lib, "pick_uv" + form)(
        u, v, ur, vr, yr, prm, uvp, q, qm, mt_lib.coef_costs(mt_lib.coef_cdfs_default(qctx, n, n, 1)),
        mt_lib.uv_mode_costs(mt_lib.uv_mode_cdfs_default()), jobs, want_cf=True, want_rec=True)
    want = getattr(oracle_lib, "pick_uv" + form)(
        u, v, ur, vr, yr, prm, uvp, q, qm, oracle_lib.default_cdfs(qctx, n, plane=1), oracle_lib.uv_mode_cdfs(), jobs,
        threads=os.cpu_count() or 1, want_cf=True, want_rec=True)
    for a, b in zip(got, want):
        assert np.asarray(a).tobytes() == np.asarray(b).tobytes()
