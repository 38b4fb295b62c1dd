"""The frontend's planes are tokenised one lane per token (bitmaps of the
non-zeros in scan order); planes given by a caller go through the warp-per-item
pass. Both must write the same file: checked on an encode's own planes handed
back through cujpegxl_b200_encode_planes, at the stripe shapes where the two
could part (one to four block rows, one to 32 blocks wide, groups of one
block), with no tokens at all, and with nearly every coefficient coded."""

from __future__ import annotations

import numpy as np
import pytest

from cujpegxl_b200 import SINGLE_GROUP, Encoder
from cujpegxl_b200.synth import make_nv12
from oracle import api

from .gpu_util import device_nv12

pytestmark = pytest.mark.gpu


def _content(kind: str, w: int, h: int) -> np.ndarray:
    if kind == "flat":
        return np.full(w * h * 3 // 2, 128, np.uint8)
    if kind == "noise":
        return np.random.Generator(np.random.PCG64(w * h)).integers(0, 256, w * h * 3 // 2).astype(np.uint8)
    return make_nv12(w, h, w + h)


@pytest.mark.parametrize("w,h", [(8, 8), (32, 24), (72, 104), (256, 256), (264, 8), (264, 40), (288, 280), (520, 264)])
@pytest.mark.parametrize("kind,distance", [("flat", 1.0), ("synth", 1.0), ("synth", 6.0), ("noise", 0.02)])
def test_lane_per_token_pass_equals_warp_per_item_pass(w, h, kind, distance):
    keep, luma, chroma, lp, cp = device_nv12(_content(kind, w, h), w, h)
    with Encoder(w, h, distance, flags=SINGLE_GROUP) as enc:
        data = enc.encode_device(luma, chroma, lp, cp)
        planes = enc.read_planes()
        sc = api.scalars(distance)
        assert enc.encode_planes(planes, sc["global_scale"], sc["quant_dc"]) == data
        # And back again: the planes of the next encode are the frontend's.
        assert enc.encode_device(luma, chroma, lp, cp) == data
