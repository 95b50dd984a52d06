"""The context and the plain trellis of the lane kernels where a cost leaves the range of a float: from a
lambda on whose products overflow, no end of block has a finite cost, none may win, and the block keeps
nothing.  Bit for bit against the oracle."""
import os

import numpy as np
import pytest

from maroontree_b200 import synth

pytestmark = pytest.mark.gpu
W, H, QIDX = 160, 96, 40


def _plane(seed):
    src = synth.rgb_to_luma(synth.generate_rgb(W, H, seed))
    return src, synth.synthetic_recon(src, seed + 5)


def _same(got, want):
    for a, b in zip(got, want):
        assert np.asarray(a).tobytes() == np.asarray(b).tobytes()


LAMBDAS = [1e34, 1e36, 3e38, float("inf")]


@pytest.mark.parametrize("family", ["leaf8", "refine8", "leaf16", "refine16", "leaf32", "grid16"])
@pytest.mark.parametrize("lam0", LAMBDAS)
def test_lane_leaves_without_a_finite_cost_match_oracle(mt_lib, oracle_lib, cuda, family, lam0):
    src, rec = _plane(QIDX)
    size = int("".join(c for c in family if c.isdigit()))
    q, qm = oracle_lib.quant_new(QIDX, 8, 6), oracle_lib.qm_row(6, 0, size)
    c = oracle_lib.default_cdfs(oracle_lib.qcat(QIDX), size)
    prm = mt_lib.split16_params(W, H, trellis_lambda0=lam0, rd_lambda=20.0, band_tilt=1.9, wsse_scale=0.5,
                                tx_guard_shift=2)
    if family == "grid16":
        jobs = synth.leaf64_jobs(W, H, range(13), (0,), seed=3, grid=True)
    else:
        jobs = synth.leaf8_jobs(W, H, range(13), (0,), seed=3, n=size)
    jobs = jobs[np.random.default_rng(3).permutation(len(jobs))[:40]]
    args, oargs = (src, rec, prm, q, qm, mt_lib.coef_costs(c), jobs), (src, rec, prm, q, qm, c, jobs)
    threads = os.cpu_count() or 1
    if family == "grid16":
        _same(mt_lib.grid16_luma(*args, want_cf=True), oracle_lib.grid16_luma(*oargs, threads=threads, want_cf=True))
    elif family == "leaf32":
        _same(mt_lib.leaf32(*args, want_cf=True, want_rec=True), oracle_lib.leaf32(*oargs, threads=threads))
    else:
        refine = family.startswith("refine")
        leaf = "leaf%d" % size
        _same(getattr(mt_lib, leaf)(*args, refine=refine, want_cf=True, want_rec=True),
              getattr(oracle_lib, leaf)(*oargs, refine=refine, threads=threads))


@pytest.mark.parametrize("form", ["16_420", "32_420", "16_444", "32_444"])
@pytest.mark.parametrize("lam0", LAMBDAS)
def test_lane_chroma_without_a_finite_cost_matches_oracle(mt_lib, oracle_lib, cuda, form, lam0):
    leaf, sub = int(form[:2]), form.endswith("420")
    n = leaf // 2 if sub else leaf
    (_, yr), (u, ur), (v, vr) = _plane(QIDX), _plane(QIDX + 1), _plane(QIDX + 2)
    if sub:
        u, ur, v, vr = [np.ascontiguousarray(a[::2, ::2]) for a in (u, ur, v, vr)]
    q, qm = oracle_lib.quant_new_chroma(QIDX, 0, 0, 8, 6), oracle_lib.qm_row(6, 1, n)
    ch, cw = u.shape
    prm = mt_lib.split16_params(cw, ch, trellis_lambda0=lam0, rd_lambda=20.0, band_tilt=0.7, wsse_scale=0.5)
    uvp = mt_lib.uv16_params(W, angle_deltas=True, dir_lambda=9.0)
    if form == "16_420":
        jobs = synth.uv16_jobs(W, H, QIDX)
    elif form == "32_444":
        jobs = synth.uv32_444_jobs(W, H, QIDX)
    else:
        jobs = synth.uv16_444_jobs(W, H, QIDX, leaf=leaf)
    qctx = oracle_lib.qcat(QIDX)
    _same(getattr(mt_lib, "pick_uv" + form)(
        u, v, ur, vr, yr, prm, uvp, q, qm, mt_lib.coef_costs(mt_lib.coef_cdfs_default(qctx, n, n, 1)),
        mt_lib.uv_mode_costs(mt_lib.uv_mode_cdfs_default()), jobs, want_cf=True, want_rec=True),
        getattr(oracle_lib, "pick_uv" + form)(
        u, v, ur, vr, yr, prm, uvp, q, qm, oracle_lib.default_cdfs(qctx, n, plane=1), oracle_lib.uv_mode_cdfs(), jobs,
        threads=os.cpu_count() or 1, want_cf=True, want_rec=True))
