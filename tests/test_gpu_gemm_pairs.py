"""The palettized GEMM on pairs of CTAs against 64-bit products of the dequantised weights, where it can go wrong: one
weight row, row tiles without a partner, token tiles of every size and their remainders, one stage of K, fewer stages than
the four slots that fill them, K cut into ranges, more tiles than pairs.

Up to 32 tokens the engine mostly chooses another kernel, so there this one is also called by itself, plain and with a residual in place.

Tolerance: fp16 inputs, fp32 sums of at most 2^12 products in any order (relative 2^-24 * 2^6 on average) and one rounding to
fp16 (2^-11 at most, 2^-11 / sqrt(3) in the mean): 4e-4 of the result's norm.  Against products rounded where the kernel rounds, only sums
that fall on the other side of a rounding differ, by 2^-10 at most, and few do: 2e-4."""
import numpy as np
import pytest

import native_util
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


# ranges of K at these token counts: 1, 1, 1, 7, 6, 3, 2, 8, and more tiles than pairs
@pytest.mark.parametrize("bits", [4, 2])
@pytest.mark.parametrize("m,k", [(8, 128), (136, 256), (264, 640), (1000, 3584), (3000, 5120), (5000, 3968), (8200, 1664), (264, 8192), (20000, 640)])
def test_few_tokens_by_themselves(backend, m, k, bits):
    import torch

    h = backend.upload("gemm_pairs.alone", synth.make_payload(m, k, bits=bits, seed=m + k), m, k, bits)
    try:
        w = torch.from_numpy(backend.dequant(h).astype(np.uint16).view(np.float16).reshape(m, k)).cuda().double()
        for t in (8, 9, 31, 32):
            rng = np.random.default_rng(t)
            x = torch.from_numpy(rng.standard_normal((t, k)).astype(np.float16)).cuda()
            old = torch.from_numpy(rng.standard_normal((t, m)).astype(np.float16)).cuda()
            prod = (x.double() @ w.T).half().double()
            y = torch.full((t, m), 7.0, dtype=torch.float16, device="cuda")
            native_util.gemm_tc5(backend, h, x, y)
            assert (y.double() - prod).norm() <= 2e-4 * prod.norm(), t
            first, want = y.clone(), (prod + old.double()).half().double()
            y.fill_(7.0)
            native_util.gemm_tc5(backend, h, x, y)
            assert torch.equal(y, first), t
            y.copy_(old)
            native_util.gemm_tc5(backend, h, x, y, resid=y)
            assert (y.double() - want).norm() <= 2e-4 * want.norm(), t
    finally:
        backend.free(h)
