"""The transform selection takes costs with error bounds and falls back to the
exact passes where the bounds leave a decision open. With the stage dumps on,
the exact passes decide everything; both must give the same planes, on content
whose costs tie or nearly tie (flat, gradients, one-step dither, repeated
blocks), at the smallest and largest quanta, and on partial regions."""

from __future__ import annotations

import ctypes

import numpy as np
import pytest

from cujpegxl_b200 import SINGLE_GROUP, Encoder, _capi
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
    elif kind.startswith("noise"):
        luma = np.clip(np.round(180 + rng.normal(0, float(kind[5:]), (h, w))), 0, 255)
    elif kind.startswith("slope"):
        luma = np.clip(np.round(90 + x * 0.05 + y * 0.06 + rng.normal(0, float(kind[5:]), (h, w))), 0, 255)
    elif kind == "edges":
        luma = np.where((x // 40 + y // 24) % 2 == 0, 0, 255)
    else:
        return make_nv12(w, h, 31)
    chroma = np.full((h // 2, w), 128)
    return np.concatenate([luma.astype(np.uint8).ravel(), chroma.astype(np.uint8).ravel()])


# Up to as many tiles as the GPU has SMs a CTA of 512 threads takes one tile;
# above, one of two halves of 256 each, which map the work otherwise: 24 x 16
# tiles, and 15 x 18 and 13 x 18 (an odd column; partial regions).
@pytest.mark.parametrize("w,h", [(256, 256), (328, 200), (1480, 1000), (904, 1096), (808, 1128)])
@pytest.mark.parametrize("kind", ["flat", "gradient", "dither", "repeated", "edges", "synth", "noise1", "noise0.3", "slope0.4"])
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


@pytest.mark.parametrize("w,h", [(640, 512), (1280, 720)])  # one tile per CTA, and pairs
@pytest.mark.parametrize("kind,most", [("flat", 0.0), ("gradient", 0.0), ("synth", 0.03), ("noise4", 0.15), ("noise2", 0.15),
                                       ("noise1", 0.1), ("noise0.4", 0.1), ("slope1", 0.25), ("slope0.4", 0.3)])
def test_few_regions_pay_for_bounds_and_exact_passes(w, h, kind, most):
    """Weak noise leaves the transforms' costs closer together than on any
    other content. Bounds that add up every coefficient's error at its largest
    left 50% to 100% of these regions open (the noisy kinds), and each of those
    paid for both passes. `most`: twice to three times the shares that a
    restatement of the bounds on the CPU gives, where the region does not go to
    the exact passes at once."""
    keep, luma, chroma, lp, cp = device_nv12(_content(kind, w, h), w, h)
    counts = (ctypes.c_uint32 * 3)()
    with Encoder(w, h, 1.0) as enc:
        inp = _capi.Nv12Input(luma, chroma, lp, cp)
        _capi.check("routes", _capi.lib().cujpegxl_b200_debug_selection_routes(enc.handle, ctypes.byref(inp), counts))
    decided, left, at_once = counts
    assert decided + left + at_once == -(-w // 32) * -(-h // 32)
    assert left <= most * (decided + left + at_once), (decided, left, at_once)
    if kind in ("flat", "gradient", "synth", "noise4"):
        assert at_once <= 0.02 * (decided + left + at_once), (decided, left, at_once)
