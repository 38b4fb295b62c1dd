"""CUDA path vs the CPU restatement, through the C ABI: every integer output of
the frontend, the FP16 coefficients, the float stage dumps and the final .jxl
bytes must be bit-identical (the float arithmetic is defined operation by
operation on both sides). Where the reference-built checker is present the
file is also compared with the reference's own assembly of the same planes.
"""

from __future__ import annotations

import numpy as np
import pytest

from cujpegxl_b200 import Encoder, acsnet
from cujpegxl_b200.decode import decode_planes, psnr_y
from cujpegxl_b200.synth import make_nv12
from oracle import api

from .gpu_util import device_nv12

pytestmark = pytest.mark.gpu

CASES = [
    (512, 384, 1.0, 0),
    (264, 264, 1.0, 1),     # two AC groups per row, one partial
    (520, 392, 2.0, 2),     # partial regions, tiles and AC groups
    (1280, 720, 0.5, 3),
    (1920, 1080, 1.0, 0),   # partial colour tiles (bh = 135)
]


def _frontend_and_file(w, h, d, seed, pitch_pad=0):
    nv = make_nv12(w, h, seed)
    keep, luma, chroma, lp, cp = device_nv12(nv, w, h, w + pitch_pad, w + pitch_pad)
    with Encoder(w, h, d) as enc:
        enc.set_debug(True)
        data = enc.encode_device(luma, chroma, lp, cp)
        planes = enc.read_planes(debug=True)
    return nv, data, planes


@pytest.mark.parametrize("w,h,d,seed", CASES)
def test_frontend_bit_exact(w, h, d, seed):
    nv, _, g = _frontend_and_file(w, h, d, seed)
    o = api.frontend(nv, w, h, d, debug=True)
    np.testing.assert_array_equal(g["xyb"].view(np.uint32), o.xyb.view(np.uint32), err_msg="xyb")
    np.testing.assert_array_equal(g["sharp"].view(np.uint32), o.sharp.view(np.uint32), err_msg="sharp")
    np.testing.assert_array_equal(g["qf"], o.qf, err_msg="quant field")
    np.testing.assert_array_equal(g["acs"], o.acs, err_msg="transform selection")
    np.testing.assert_array_equal(g["coeff"], o.coeff, err_msg="fp16 coefficients")
    np.testing.assert_array_equal(g["ytox"], o.ytox, err_msg="ytox")
    np.testing.assert_array_equal(g["ytob"], o.ytob, err_msg="ytob")
    np.testing.assert_array_equal(g["ac"], o.ac, err_msg="quantised AC")
    np.testing.assert_array_equal(g["dc"], o.dc, err_msg="quantised DC")


@pytest.mark.parametrize("w,h,d,seed", CASES)
def test_file_bit_exact(w, h, d, seed):
    nv, data, g = _frontend_and_file(w, h, d, seed)
    assert data == api.encode(nv, w, h, d)
    if api.ref_available():
        r = api.FrontendResult(w, h)
        for k in ("ac", "dc", "acs", "qf", "ytox", "ytob"):
            getattr(r, k)[...] = g[k]
        assert data == api.ref_encode_frame(r, d)


@pytest.mark.parametrize("d", [0.5, 1.0, 2.0, 4.0])
def test_4k_file_and_planes_bit_exact(d):
    """The benchmark frame at every distance of the 4K configuration: the
    quantised planes and the file equal the CPU restatement's."""
    w, h = 3840, 2160
    nv = make_nv12(w, h, 0)
    keep, luma, chroma, lp, cp = device_nv12(nv, w, h)
    with Encoder(w, h, d) as enc:
        data = enc.encode_device(luma, chroma, lp, cp)
        g = enc.read_planes()
    o = api.frontend(nv, w, h, d)
    for k in ("qf", "acs", "ytox", "ytob", "ac", "dc"):
        np.testing.assert_array_equal(g[k], getattr(o, k), err_msg=k)
    assert data == api.encode(nv, w, h, d)
    # Full-size round trip through the in-repo decoder: the file holds exactly
    # the planes the GPU computed.
    back = decode_planes(data)
    first = g["acs"] != 0
    for k in ("acs", "dc", "ytox", "ytob", "ac"):
        np.testing.assert_array_equal(back[k], g[k], err_msg=f"decoded {k}")
    np.testing.assert_array_equal(back["qf"][first], g["qf"][first])


def test_4k_quality_falls_with_distance():
    w, h = 3840, 2160
    nv = make_nv12(w, h, 0)
    keep, luma, chroma, lp, cp = device_nv12(nv, w, h)
    psnr = []
    with Encoder(w, h, 0.5) as enc:
        for d in (0.5, 1.0, 2.0, 4.0):
            enc.configure(w, h, d)
            psnr.append(psnr_y(nv, enc.encode_device(luma, chroma, lp, cp)))
    assert all(a > b for a, b in zip(psnr, psnr[1:])), psnr
    assert psnr[1] > 40.0, psnr


def test_pitched_input_matches_packed():
    w, h = 512, 384
    _, packed, _ = _frontend_and_file(w, h, 1.0, 5)
    _, pitched, _ = _frontend_and_file(w, h, 1.0, 5, pitch_pad=96)
    assert packed == pitched


def test_deterministic_and_reusable():
    w, h = 640, 384
    nv = make_nv12(w, h, 11)
    keep, luma, chroma, lp, cp = device_nv12(nv, w, h)
    with Encoder(w, h, 1.0) as enc:
        a = enc.encode_device(luma, chroma, lp, cp)
        b = enc.encode_device(luma, chroma, lp, cp)
        enc.configure(w, h, 2.0)
        c = enc.encode_device(luma, chroma, lp, cp)
    assert a == b
    assert c == api.encode(nv, w, h, 2.0)


def test_host_input_path_matches_device_path():
    w, h = 512, 512
    nv = make_nv12(w, h, 3)
    keep, luma, chroma, lp, cp = device_nv12(nv, w, h)
    with Encoder(w, h, 1.0) as enc:
        a = enc.encode_device(luma, chroma, lp, cp)
        b = enc.encode_host(nv)
    assert a == b


# Frames of more tiles than the GPU has SMs take two tiles per CTA: 15 x 18 and
# 13 x 18 tiles (an odd column, whose right half leaves at once, and partial
# regions on both sides). Without the stage dumps, so that the bounds decide.
@pytest.mark.parametrize("network", [False, True])
@pytest.mark.parametrize("w,h,d", [(904, 1096, 1.0), (808, 1128, 0.4), (1480, 1000, 3.0)])
def test_paired_tiles_file_bit_exact(w, h, d, network):
    """Against the restatement. With an all-zero network, which decides
    nothing, the tiles come in the order that the inference kernel writes."""
    nv = make_nv12(w, h, 7)
    keep, luma, chroma, lp, cp = device_nv12(nv, w, h)
    with Encoder(w, h, d) as enc:
        if network:
            norm = np.array([30.0, 4.0, 4.0, 1.0, 0.0, 0.4, 0.4, 0.5], np.float32)
            net = acsnet.AcsNet(acsnet.pack_blob(np.zeros(acsnet.NPARAMS, np.float32), norm))
            enc.set_acsnet(net, 0.2, acsnet.SPLIT | acsnet.QF)
        assert enc.encode_device(luma, chroma, lp, cp) == api.encode(nv, w, h, d)


def test_more_sections_than_layout_threads_bit_exact():
    """1161 sections (1030 AC and 129 DC groups of a column of blocks): the
    threads of the layout's one block take two TOC entries each."""
    w, h, d = 8, 1030 * 256, 1.0
    rng = np.random.Generator(np.random.PCG64(8))
    luma8 = np.repeat(rng.integers(0, 256, (h // 4, w // 2)), 4, axis=0).repeat(2, axis=1)
    nv = np.concatenate([luma8.ravel(), np.full(w * h // 2, 128)]).astype(np.uint8)
    keep, luma, chroma, lp, cp = device_nv12(nv, w, h)
    with Encoder(w, h, d) as enc:
        assert enc.encode_device(luma, chroma, lp, cp) == api.encode(nv, w, h, d)


TOKENS_PER_BLOCK = 32  # places of a block in the token pool


def _tokens(g: dict) -> int:
    """AC tokens of a frame's planes: a count per first block and channel, and
    every scan position through the last non-zero coefficient, here at least
    the non-zeros."""
    first = int((g["acs"] != 0).sum())
    return 3 * first + int((g["ac"] != 0).sum())


def test_tokens_beyond_their_places_bit_exact():
    """At distance 0.05 a 520x392 frame has more AC tokens than the pool has
    places: those of the frontend's own planes go to the unused end of the
    output buffer. Still the restatement's file."""
    w, h, d = 520, 392, 0.05
    nv, data, g = _frontend_and_file(w, h, d, 2)
    assert _tokens(g) > TOKENS_PER_BLOCK * (w // 8) * (h // 8)
    assert data == api.encode(nv, w, h, d)


def test_token_pool_overflow_of_given_planes_bit_exact():
    """The same planes given by the caller: the stripes that find the pool full
    are tokenised again from their coefficients in the length and emission
    passes (planes from a frontend never are)."""
    w, h, d = 520, 392, 0.05
    nv, data, g = _frontend_and_file(w, h, d, 2)
    assert _tokens(g) > TOKENS_PER_BLOCK * (w // 8) * (h // 8)
    sc = api.scalars(d)
    with Encoder(w, h, d) as enc:
        given = enc.encode_planes({k: g[k] for k in ("ac", "dc", "acs", "qf", "ytox", "ytob")}, sc["global_scale"],
                                  sc["quant_dc"])
    assert given == api.encode(nv, w, h, d)
