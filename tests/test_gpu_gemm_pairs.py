"""The palettized GEMM on pairs of CTAs against 64-bit products of the dequantised weights, where it can go wrong: one
weight row, row tiles without a partner, token tiles of every size and their remainders, one stage of K, fewer stages than
the four slots that fill them, K cut into ranges, more tiles than pairs.

Tolerance: fp16 inputs, fp32 sums of at most 2^12 products in any order (relative 2^-24 * 2^6 on average) and one rounding to
fp16 (2^-11 at most, 2^-11 / sqrt(3) in the mean): 4e-4 of the result's norm."""
import numpy as np
import pytest

from prism_engine_b200 import synth

pytestmark = pytest.mark.gpu


def _check(backend, m, k, bits, tokens):
    name = "gemm_pairs.%d.%d.%d" % (m, k, bits)
    h = backend.upload(name, synth.make_payload(m, k, bits=bits, seed=m + k), m, k, bits)
    w = backend.dequant(h).astype(np.uint16).view(np.float16).astype(np.float64).reshape(m, k)
    try:
        for t in tokens:
            x = (np.random.default_rng(t).standard_normal((t, k))).astype(np.float16)
            got = np.asarray(backend.gemm(h, x.view(np.uint16))).view(np.float16).astype(np.float64)
            want = x.astype(np.float64) @ w.T
            assert np.linalg.norm(got - want) <= 4e-4 * np.linalg.norm(want), (t, np.linalg.norm(got - want) / np.linalg.norm(want))
            again = np.asarray(backend.gemm(h, x.view(np.uint16))).view(np.float16).astype(np.float64)
            assert np.array_equal(got, again), t
    finally:
        backend.free(h)


@pytest.mark.parametrize("bits", [4, 2])
@pytest.mark.parametrize("m,k", [(8, 128), (136, 256), (264, 640), (1000, 3584)])
def test_tiles_and_ranges(backend, m, k, bits):
    _check(backend, m, k, bits, (8, 9, 31, 32, 33, 64, 65, 129, 192, 255, 257, 300))


@pytest.mark.parametrize("bits", [4, 2])
def test_more_tiles_than_pairs(backend, bits):
    _check(backend, 4104, 384, bits, (1300,))
    _check(backend, 20000, 128, bits, (16, 300))
