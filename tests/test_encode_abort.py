"""The end of the decision kernel's waits: a frame whose first block nobody codes, so that every other block
waits for records that nothing writes.  The call returns the device error after the waits' limit, with all
clusters gone, and the next encode is whole: with a cluster for every runnable block (late tickets), with
fewer (early ones), and with more blocks than clusters."""
import ctypes as C

import numpy as np
import pytest

from maroontree_b200 import abi, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,chroma", [(16, 8, 0), (136, 72, 0), (512, 512, 2), (2304, 2304, 0)])
def test_waits_that_run_out_end_the_call_with_an_error(mt_lib, cuda, w, h, chroma):
    from maroontree_b200 import encoder as enc

    lib = mt_lib.load()
    call = lib._ZN3mth26encode_without_first_blockEPKhjjPK16mt_encode_config
    call.restype, call.argtypes = C.c_int, (C.c_void_p, C.c_uint32, C.c_uint32, C.c_void_p)
    rgb, cfg = synth.generate_rgb(w, h, 7), enc.config(quality=60, chroma=chroma)
    before = enc.encode_rgb8(rgb, cfg)
    assert call(np.ascontiguousarray(rgb).ctypes.data, w, h, C.addressof(cfg)) == abi.MT_ERR_DEVICE
    assert enc.encode_rgb8(rgb, cfg) == before
