"""The 8x8 level with eight lanes per candidate at the edges of what it takes,
and the calls it leaves to the thread-per-candidate kernel, bit for bit against
the oracle: fewer blocks than a warp has groups, positions off the 8-sample
grid, every transform type, full-scale residuals at the smallest steps (levels
past 63, Golomb remainders), no trellis, skip prices, a cut display, a
quantiser whose multiplier passes 16 bits."""
import numpy as np
import pytest

from maroontree_b200 import abi, synth

pytestmark = pytest.mark.gpu

CASES = [
    # blocks, offset, qidx, qm_level, lambda0, options
    (1, 0, 70, 6, 0.05, ()), (3, 3, 116, 1, 0.05, ()), (5, 0, 4, 15, 0.05, ("extreme",)),
    (17, 5, 1, 8, 0.4, ("extreme", "vis")), (9, 0, 200, 15, 0.0, ("skip",)), (33, 1, 30, 4, 0.05, ("untrellised", "skip")),
    (6, 2, 90, 6, 0.05, ("general",)), (7, 0, 1, 15, 0.05, ("general", "extreme")),
]


@pytest.mark.parametrize("nblocks,offset,qidx,qm_level,lambda0,options", CASES)
def test_level_matches_oracle(mt_lib, oracle_lib, cuda, nblocks, offset, qidx, qm_level, lambda0, options):
    import maroontree_b200 as mt

    w, h = 96, 72
    rng = np.random.default_rng(nblocks)
    src = synth.rgb_to_luma(synth.generate_rgb(w, h, qidx))
    rec = synth.synthetic_recon(src, qidx + 7)
    if "extreme" in options:
        src = np.where(rng.random((h, w)) < 0.5, 0, 255).astype(np.uint16)
        rec = (255 - src).astype(np.uint16)
    blocks = synth.level_blocks(w, h, seed=qidx)[:nblocks].copy()
    blocks["px"] = np.minimum(blocks["px"] + offset, w - 8)
    blocks["py"] = np.minimum(blocks["py"] + offset, h - 8)
    combos = synth.level_combos(range(13), range(7), (-2, 0), delta_bits=lambda m, d: 0.25 + 0.1 * m)
    if "untrellised" in options:
        combos["flags"][::3] |= abi.COMBO_NO_TRELLIS
    q = oracle_lib.quant_new(qidx, 8, qm_level)
    if "general" in options:
        q.q_mult_dc = 40000
    qm = oracle_lib.qm_row(qm_level, 0, 8)
    cdfs = synth.synthetic_cdfs(qidx + 1)
    prm = mt.chain_params(w, h, trellis_lambda0=lambda0, mode_lambda=0.3 * qidx + 2.0, satd_scale=1.25,
                          satd_bridge=0.8, **({"skip_bits": (0.7, 1.9)} if "skip" in options else {}))
    if "vis" in options:
        prm.vis_w, prm.vis_h = w - 5, h - 3
    best, res = mt_lib.rdo_level8(src, rec, prm, q, qm, mt_lib.coef_costs(cdfs), blocks, combos, want_results=True)
    ref, _, _ = oracle_lib.candidate_chain(src, rec, prm, q, qm, cdfs, synth.candidates_of_level(blocks, combos),
                                           threads=8)
    assert res.tobytes() == ref.tobytes()
    assert np.array_equal(best["combo"], synth.best_of_level(ref, len(blocks), len(combos)))
