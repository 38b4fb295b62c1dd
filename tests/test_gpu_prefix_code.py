"""The device prefix-code builder (the warp-cooperative construction every
encode runs: one merge per count floor on every lane, canonical codes and the
code-length-code header written across the warp) against the reference's
own build_and_store_huffman_tree outputs in tests/golden/huffman.npz: 27
histograms from one to 256 symbols, Fibonacci counts that force the 15-bit
depth limit, sparse and dense random cases. Depths, codes, header bits and
header length must all be equal."""

from __future__ import annotations

import ctypes
from pathlib import Path

import numpy as np
import pytest

from cujpegxl_b200 import _capi
from oracle import api

pytestmark = pytest.mark.gpu

GOLD = Path(__file__).resolve().parent / "golden" / "huffman.npz"


def _device_code(h: np.ndarray):
    depth = np.zeros(h.size, np.uint8)
    bits = np.zeros(h.size, np.uint16)
    head = np.zeros(256, np.uint8)
    nbits = ctypes.c_uint32(0)
    assert _capi.lib().cujpegxl_b200_debug_prefix_code(0, h.ctypes.data, h.size, depth.ctypes.data, bits.ctypes.data,
                                                       head.ctypes.data, head.size, ctypes.byref(nbits)) == _capi.OK
    return depth, bits, head[: (nbits.value + 7) // 8], nbits.value


@pytest.mark.parametrize("length", [2, 3, 4, 5, 33, 254, 255, 256])
@pytest.mark.parametrize("kind", ["largest", "even", "steep"])
def test_device_prefix_codes_equal_serial_builder(length, kind):
    """Alphabets around whole vectors of four counts, one of them the largest
    32-bit count ("largest"; the others' sum stays below it), and lengths whose
    symbols lie in every round of 32 ("even", "steep")."""
    rng = np.random.Generator(np.random.PCG64(length))
    h = np.ones(length, np.uint32) if kind == "even" else rng.integers(1, 50, length).astype(np.uint32)
    if kind == "largest":
        h[length // 2] = 0xFFFFFFFF
    elif kind == "steep":
        h[rng.integers(0, length, min(length, 20))] = 1 << np.arange(min(length, 20))
    depth = np.zeros(length, np.uint8)
    bits = np.zeros(length, np.uint16)
    head = np.zeros(512, np.uint8)
    nbits = api.oracle().oracle_huffman(h.ctypes.data, length, depth.ctypes.data, bits.ctypes.data, head.ctypes.data, 512)
    got = _device_code(h)
    assert got[3] == nbits
    np.testing.assert_array_equal(got[0], depth)
    np.testing.assert_array_equal(got[1], bits)
    np.testing.assert_array_equal(got[2], head[: (nbits + 7) // 8])


def test_device_prefix_codes_equal_reference_golden():
    z = np.load(GOLD)
    L = _capi.lib()
    i = 0
    limited = 0
    while f"hist{i}" in z:
        h = np.ascontiguousarray(z[f"hist{i}"].astype(np.uint32))
        depth = np.zeros(h.size, np.uint8)
        bits = np.zeros(h.size, np.uint16)
        head = np.zeros(256, np.uint8)
        nbits = ctypes.c_uint32(0)
        code = L.cujpegxl_b200_debug_prefix_code(0, h.ctypes.data, h.size, depth.ctypes.data, bits.ctypes.data,
                                                 head.ctypes.data, head.size, ctypes.byref(nbits))
        assert code == _capi.OK, i
        np.testing.assert_array_equal(depth, z[f"depth{i}"], err_msg=f"case {i}")
        np.testing.assert_array_equal(bits, z[f"bits{i}"], err_msg=f"case {i}")
        assert nbits.value == int(z[f"nbits{i}"][0]), i
        np.testing.assert_array_equal(head[: (nbits.value + 7) // 8], z[f"header{i}"], err_msg=f"case {i}")
        limited += int(depth.max() == 15)
        i += 1
    assert i > 20 and limited >= 1
