"""mt_encode_rgb8_batch away from device 0.  A batch finishes its images on
threads of its own, which start on device 0: they have to work on the caller's
device, whose streams and buffers they use."""
import pytest

from maroontree_b200 import synth

pytestmark = pytest.mark.gpu


def test_batch_encode_on_another_device(mt_lib, cuda):
    from maroontree_b200 import encoder as enc

    if cuda.cuda.device_count() < 2:
        pytest.skip("needs two CUDA devices")
    imgs = [synth.generate_rgb(w, h, 40 + w) for w, h in ((136, 72), (200, 136))]
    cfg = enc.config(quality=60)
    want = [enc.encode_rgb8(im, cfg) for im in imgs]
    with cuda.cuda.device(1):
        assert enc.encode_rgb8_batch(imgs, cfg) == want
        # the buffers that the batch grew serve single calls
        assert [enc.encode_rgb8(im, cfg) for im in imgs] == want
        mt_lib.load().mt_encode_release_buffers()
