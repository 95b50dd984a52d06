"""The 8x8 leaf searches with eight lanes per job: job counts around a warp's
and a CTA's blocks, rejected jobs among good ones, every transform type of the
refinement (the 1-D walk of V_DCT and H_DCT among them), cut displays, levels of
every size class, no trellis.  Bit for bit against the oracle."""
import os

import numpy as np
import pytest

from maroontree_b200 import synth

pytestmark = pytest.mark.gpu
W, H = 176, 88


def _planes(kind, seed):
    rng = np.random.default_rng(seed)
    if kind == "flat":
        src = (80 + rng.integers(0, 3, (H, W))).astype(np.uint16)
    elif kind == "hard":
        src = np.where(rng.random((H, W)) < 0.5, 0, 255).astype(np.uint16)
    elif kind == "lines":  # one direction constant: the one-pass types win
        src = np.repeat(rng.integers(0, 256, (1, W)), H, 0).astype(np.uint16)
    else:
        src = synth.rgb_to_luma(synth.generate_rgb(W, H, seed))
    return src, synth.synthetic_recon(src, seed + 5)


@pytest.mark.parametrize("form", ["modes", "refine", "refine_all"])
@pytest.mark.parametrize("n,kind,qidx,vis,wsse,lam0", [
    (1, "photo", 70, None, 0.0, 0.05), (3, "hard", 1, (171, 83), 1.0, 0.05), (31, "flat", 200, (169, 81), 0.5, 0.3),
    (33, "lines", 40, (170, 84), 1.0, 0.0), (70, "lines", 10, None, 0.0, 0.05), (97, "photo", 140, (173, 85), 1.0, 0.2)])
def test_leaf8_matches_oracle(mt_lib, oracle_lib, cuda, form, n, kind, qidx, vis, wsse, lam0):
    src, rec = _planes(kind, qidx + n)
    qm_level = 15 if qidx == 1 else 4 + qidx % 9
    q = oracle_lib.quant_new(qidx, 8, qm_level)
    qm = oracle_lib.qm_row(qm_level, 0, 8) if qm_level < 15 else None
    c = oracle_lib.default_cdfs(oracle_lib.qcat(qidx), 8)
    jobs = synth.leaf8_jobs(W, H, range(13), (-2, 0, 3), seed=n, n=8)
    jobs = jobs[np.random.default_rng(n).permutation(len(jobs))[:n]]
    for i in range(2, n, 5):  # rejected: outside the frame, or no such mode
        jobs["mode" if i % 2 else "px"][i] = 13 if i % 2 else W - 4
    prm = mt_lib.split16_params(W, H, trellis_lambda0=lam0, rd_lambda=0.02 if kind == "hard" else 0.5 * qidx + 1.0,
                                band_tilt=1.9 if n % 2 else 0.0, wsse_scale=wsse, tx_search=form == "refine_all",
                                tx_guard_shift=2, vis=vis,
                                skip_bits=[(2.5 + k, 0.4) for k in range(13)] if n % 3 else None)
    refine = form != "modes"
    got = mt_lib.leaf8(src, rec, prm, q, qm, mt_lib.coef_costs(c), jobs, refine=refine, want_cf=True, want_rec=True)
    want = oracle_lib.leaf8(src, rec, prm, q, qm, c, jobs, refine=refine, threads=os.cpu_count() or 1)
    for a, b in zip(got, want):
        assert np.asarray(a).tobytes() == np.asarray(b).tobytes()
