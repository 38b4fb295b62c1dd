"""The transform selection takes costs with error bounds and falls back to the
exact passes where the bounds leave a decision open. With the stage dumps on,
the exact passes decide everything; both must give the same planes, on content
whose costs tie or nearly tie (flat, gradients, one-step dither, repeated
blocks), at the smallest and largest quanta, and on partial regions."""

from __future__ import annotations

import numpy as np
import pytest

from cujpegxl_b200 import SINGLE_GROUP, Encoder
from cujpegxl_b200.synth import make_nv12

from .gpu_util import device_nv12

pytestmark = pytest.mark.gpu


def _content(kind: str, w: int, h: int) -> np.ndarray:
    rng = np.random.Generator(np.random.PCG64(w + h))
    y, x = np.mgrid[0:h, 0:w]
    if kind == "flat":
        luma = np.full((h, w), 200)
    elif kind == "gradient":
        luma = (x * 0.21 + y * 0.13) % 256
    elif kind == "dither":
        luma = 90 + (rng.random((h, w)) < 0.5)
    elif kind == "repeated":
        luma = np.tile(rng.integers(0, 256, (8, 8)), (h // 8, w // 8))
    elif kind == "edges":
        luma = np.where((x // 40 + y // 24) % 2 == 0, 0, 255)
    else:
        return make_nv12(w, h, 31)
    chroma = np.full((h // 2, w), 128)
    return np.concatenate([luma.astype(np.uint8).ravel(), chroma.astype(np.uint8).ravel()])


@pytest.mark.parametrize("w,h", [(256, 256), (328, 200)])
@pytest.mark.parametrize("kind", ["flat", "gradient", "dither", "repeated", "edges", "synth"])
@pytest.mark.parametrize("distance", [0.01, 0.5, 1.0, 9.0])
def test_bounded_selection_decides_as_the_exact_passes(w, h, kind, distance):
    keep, luma, chroma, lp, cp = device_nv12(_content(kind, w, h), w, h)
    planes = []
    for exact in (False, True):
        with Encoder(w, h, distance, flags=SINGLE_GROUP) as enc:
            enc.set_debug(exact)
            enc.encode_device(luma, chroma, lp, cp)
            planes.append(enc.read_planes())
    for key in planes[0]:
        assert np.array_equal(planes[0][key], planes[1][key]), key
