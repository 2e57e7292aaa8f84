"""The palettized linear of few tokens with palettes in registers, by itself against 64-bit products rounded where the kernel rounds:
rows and k that leave chunks, octets and jobs unfilled, clusters of every size, rows of y apart or not 16-byte aligned, infinite
entries that no weight uses.

Tolerance: as for the other GEMMs, values whose fp32 sum (at most 2^15 products) falls on the other side of a rounding differ by one
unit, at most 2^-10 of a value; few do: 2e-4 of the norm."""
import numpy as np
import pytest

import native_util
from prism_engine_b200 import synth

pytestmark = pytest.mark.gpu
SHAPES = {4: [(8, 32), (33, 96), (130, 160), (1000, 896), (896, 4864), (4608, 3584), (3584, 18944)],
          2: [(8, 64), (33, 192), (130, 320), (1000, 896), (896, 4864), (4608, 3584), (3584, 18944)]}


def _upload(backend, name, m, k, bits, seed):
    import torch

    h = backend.upload(name, synth.make_payload(m, k, bits=bits, seed=seed), m, k, bits)
    return h, torch.from_numpy(backend.dequant(h).astype(np.uint16).view(np.float16).astype(np.float64).reshape(m, k)).cuda()


def _rows(t, n, apart, seed):
    import torch

    x = torch.from_numpy(np.random.default_rng(seed).standard_normal((t, n + apart)).astype(np.float16)).cuda()
    return x[:, :n]


def _close(got, want):
    assert bool((got.double() - want).norm() <= 2e-4 * want.norm()), float((got.double() - want).norm() / want.norm())


@pytest.mark.parametrize("bits,m,k", [(b, *s) for b in SHAPES for s in SHAPES[b]])
def test_products(backend, bits, m, k):
    import torch

    gate, wg = _upload(backend, "gate", m, k, bits, m + k)
    up, wu = _upload(backend, "up", m, k, bits, m + k + 1)
    try:
        for t in (1, 2, 7, 8, 9, 16, 17, 24, 25, 32):
            if m == 3584 and t > 16:
                continue  # the longest part of X of this shape does not fit beside the sums
            x = _rows(t, k, 8 if t % 2 else 0, t)
            prod = (x.double() @ wg.T).half().double()
            y = torch.zeros(t, m + (8 if t % 3 else 3), dtype=torch.float16, device="cuda")
            native_util.linear_few_tokens(backend, gate, x, y[:, :m])
            _close(y[:, :m], prod)
            assert bool((y[:, m:] == 0).all())
            h = _rows(t, m, 0, t + 1).clone()
            want = (prod + h.double()).half().double()
            again = h.clone()
            native_util.linear_few_tokens(backend, gate, x, h, resid=h)
            _close(h, want)
            native_util.linear_few_tokens(backend, gate, x, again, resid=again)
            assert torch.equal(h, again), t
            if m * k < 1 << 25:
                u = (x.double() @ wu.T).half().double()
                out = torch.empty(t, m, dtype=torch.float16, device="cuda")
                native_util.linear_few_tokens(backend, gate, x, out, up=up)
                _close(out, ((prod / (1.0 + (-prod).exp())).half().double() * u).half().double())
        x = _rows(1, k, 0, 5)
        scale = (x.double().square().mean() + 1e-5).rsqrt()
        y = torch.empty(1, m, dtype=torch.float16, device="cuda")
        native_util.linear_few_tokens(backend, gate, x, y, norm_eps=1e-5)
        _close(y, ((x.double() * scale).half().double() @ wg.T).half().double())
    finally:
        backend.free(gate)
        backend.free(up)


@pytest.mark.parametrize("bits,k", [(4, 32), (4, 160), (2, 64), (2, 320)])
def test_entries_that_no_weight_uses_do_not_count(backend, bits, k):
    import torch

    m, n = 40, 1 << bits
    rng = np.random.default_rng(k)
    pal = rng.standard_normal((m, n)).astype(np.float16)
    pal[:, 0] = np.inf  # entry 0 is what lies behind the end of a row
    pal[:, 1] = np.nan
    idx = rng.integers(2, n, size=(m, k))
    packed = np.zeros((m, k * bits // 8), np.uint8)
    for j in range(8 // bits):
        packed |= (idx[:, j::8 // bits] << (j * bits)).astype(np.uint8)
    handle = backend.upload("unused", np.concatenate([pal.view(np.uint8).reshape(-1), packed.reshape(-1)]), m, k, bits)
    try:
        w = torch.from_numpy(np.take_along_axis(pal, idx, 1).astype(np.float64)).cuda()
        x = _rows(3, k, 0, 1)
        y = torch.empty(3, m, dtype=torch.float16, device="cuda")
        native_util.linear_few_tokens(backend, handle, x, y)
        _close(y, (x.double() @ w.T).half().double())
    finally:
        backend.free(handle)
