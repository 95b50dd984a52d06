"""The CDEF strength search on both of its paths: one cluster (up to 943 64x64
units) and the chain of launches (more), against the oracle's decision, grid
and filtered planes; one unit, fewer units than a warp has lanes, the last
count of the first path and the first frame of the second."""
import numpy as np
import pytest

from maroontree_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,sub,mono,q,slow,seed", [
    (8, 8, (1, 1), False, 90, True, 1), (40, 24, (0, 0), False, 220, False, 2), (700, 200, (1, 1), True, 40, False, 3),
    (1472, 2624, (1, 1), False, 60, True, 4), (1536, 2560, (1, 1), False, 60, True, 5)])
def test_search_matches_oracle(mt_lib, oracle_lib, cuda, w, h, sub, mono, q, slow, seed):
    src, rec, skip = synth.cdef_inputs(w, h, sub[0], sub[1], mono, seed)
    prm = mt_lib.cdef_params(w, h, sub[0], sub[1], q, mono=mono, slow=slow)
    want_planes, want, _ = oracle_lib.cdef_frame(rec, src, skip, prm)
    got_planes, got = mt_lib.cdef_frame(rec, src, skip, prm)
    assert (got["bits"], got["strengths"]) == (want["bits"], want["strengths"])
    assert np.array_equal(got["grid"], want["grid"])
    for a, b in zip(got_planes, want_planes):
        assert np.array_equal(a, b)
