"""What the palettized GEMM does on the way out -- the residual added, silu(gate) * up -- by itself against 64-bit products rounded
where the kernel rounds: K cut into ranges, tiles without a partner, remainders of rows and tokens, rows of a length that
the wide stores cannot take (two kernels then).

Tolerance: the rounded products differ from the exact ones' rounding in few values (fp32 sums of at most 2^12 products); where
they do it is one unit, at most 2^-10 of a value: 2e-4 of the norm."""
import numpy as np
import pytest

import native_util
from prism_engine_b200 import synth

pytestmark = pytest.mark.gpu
TOKENS = (8, 9, 31, 33, 64, 129, 257, 300)


def _upload(backend, name, m, k, bits, seed):
    import torch

    h = backend.upload(name, synth.make_payload(m, k, bits=bits, seed=seed), m, k, bits)
    return h, torch.from_numpy(backend.dequant(h).astype(np.uint16).view(np.float16).astype(np.float64).reshape(m, k)).cuda()


def _x(t, k):
    import torch

    return torch.from_numpy(np.random.default_rng(t).standard_normal((t, k)).astype(np.float16)).cuda()


def _close(got, want):
    err = (got.double() - want).norm() / want.norm()
    assert err <= 2e-4, float(err)


@pytest.mark.parametrize("bits", [4, 2])
@pytest.mark.parametrize("m,k", [(8, 128), (136, 256), (264, 640), (1000, 3584), (130, 512)])
def test_residual(backend, m, k, bits):
    import torch

    handle, w = _upload(backend, "epilogue", m, k, bits, m + k)
    try:
        for t in TOKENS:
            x, h = _x(t, k), _x(t + 1, m)[:t].clone()
            want = ((x.double() @ w.T).half().double() + h.double()).half().double()
            again = h.clone()
            native_util.gemm_add(backend, handle, x, h)
            _close(h, want)
            native_util.gemm_add(backend, handle, x, again)
            assert torch.equal(h, again), t
    finally:
        backend.free(handle)


@pytest.mark.parametrize("bits", [4, 2])
@pytest.mark.parametrize("m,k", [(8, 128), (136, 256), (264, 640), (1000, 3584), (130, 512)])
def test_swiglu(backend, m, k, bits):
    import torch

    gate, wg = _upload(backend, "gate", m, k, bits, m + k)
    up, wu = _upload(backend, "up", m, k, bits, m + k + 1)
    try:
        for t in TOKENS:
            x = _x(t, k)
            g, u = (x.double() @ wg.T).half().double(), (x.double() @ wu.T).half().double()
            want = ((g / (1.0 + (-g).exp())).half().double() * u).half().double()
            for fused in (False, True) if m % 8 == 0 else (False,):
                out = torch.empty(t, m, dtype=torch.float16, device="cuda")
                native_util.gemm_swiglu(backend, gate, up, x, out, fused)
                _close(out, want)
    finally:
        backend.free(gate)
        backend.free(up)
