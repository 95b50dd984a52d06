"""The encoder's entropy coding on the device at the edges of its pieces: one
block, a flat picture (long runs of each CDF's first symbol, whole pieces with
no store to start from), noise at high quality (Golomb remainders, 16-bit
renormalisations), a token count just over a group of pieces, two tiles.  The
file equals the oracle encode's byte for byte; without CDF adaptation the
decoder's picture equals the encoder's reconstruction."""
import io

import numpy as np
import pytest

from maroontree_b200 import synth

pytestmark = pytest.mark.gpu


def _picture(kind, w, h):
    rng = np.random.default_rng(w * 7 + h)
    if kind == "flat":
        return np.full((h, w, 3), 93, np.uint8)
    if kind == "noise":
        return rng.integers(0, 256, (h, w, 3), dtype=np.uint8)
    if kind == "bars":
        x = (np.arange(w) // 3 % 2 * 255).astype(np.uint8)
        return np.repeat(np.repeat(x[None, :, None], h, 0), 3, 2)
    return synth.generate_rgb(w, h, 5)


@pytest.mark.parametrize("kind,w,h,quality,chroma", [
    ("plain", 8, 8, 60, 0), ("plain", 1, 1, 60, 2), ("flat", 8, 8, 1, 2), ("flat", 1024, 512, 50, 0),
    ("flat", 264, 200, 99, 2), ("noise", 96, 72, 97, 2), ("noise", 200, 64, 90, 0), ("bars", 136, 136, 85, 2),
    ("plain", 64, 64, 30, 0), ("plain", 65, 129, 70, 2), ("noise", 4168, 16, 60, 0), ("flat", 4168, 72, 60, 2)])
def test_device_coded_file_equals_the_oracle(mt_lib, oracle_lib, cuda, kind, w, h, quality, chroma):
    from maroontree_b200 import encoder as enc
    from oracle import oracle_avif as oa

    rgb = _picture(kind, w, h)
    assert enc.encode_rgb8(rgb, enc.config(quality=quality, chroma=chroma)) == oa.encode_rgb8(rgb, quality, chroma)


@pytest.mark.parametrize("kind,w,h,quality", [("plain", 72, 136, 60), ("noise", 64, 64, 95), ("flat", 128, 64, 40)])
def test_without_adaptation_the_decoder_gets_the_reconstruction(mt_lib, cuda, kind, w, h, quality):
    from PIL import Image

    from maroontree_b200 import encoder as enc

    rgb = _picture(kind, w, h)
    avif, rec = enc.encode_yuv8(rgb[..., 1], rgb[..., 2], rgb[..., 0],
                                enc.config(quality=quality, chroma=2, matrix=0, updating_cdf=0), want_recon=True)
    dec = np.asarray(Image.open(io.BytesIO(avif)).convert("RGB"))
    for plane, channel in ((0, 1), (1, 2), (2, 0)):
        assert np.array_equal(dec[..., channel], rec[plane][:h, :w])
