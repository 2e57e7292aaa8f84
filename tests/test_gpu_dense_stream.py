"""The streaming dense linear of few rows against 64-bit products: row tiles with few valid rows, one and many CTAs a tile, segments of
other lengths and inputs (equal ranges of all units then), activations, bias and stores; repeated calls give the same bits and leave
the arrival counters as they were.

Tolerance: bf16 results, rounded once from fp32 sums: bf16 keeps 8 bits, so at most 2^-8 of a value, 3.91e-3 (reached where there is one
row of one value): 4e-3 of the norm; fp32 results 1e-5."""
import pytest

import native_util

pytestmark = pytest.mark.gpu


def _bf16(rows, cols, seed, scale=1.0):
    import torch

    g = torch.Generator(device="cuda").manual_seed(seed)
    return (torch.randn(rows, cols, device="cuda", generator=g) * scale).bfloat16()


def _close(got, want, tol):
    err = float((got.double() - want).norm() / want.norm())
    assert err <= tol, err


@pytest.mark.parametrize("rows,k", [(128, 64), (1, 64), (130, 128), (37, 4096), (896, 5760), (3000, 1536), (20000, 640), (37900, 192), (40000, 128)])
def test_one_segment(backend, rows, k):
    import torch

    tiles = (rows + 127) // 128
    w = torch.zeros(tiles * 128, k, dtype=torch.bfloat16, device="cuda")
    w[:rows] = _bf16(rows, k, rows)
    packed = native_util.dense_layout(w)
    for t in (1, 2, 5, 8):
        x = _bf16(t, k + 64, t)[:, :k]
        want = x.double() @ w[:rows].double().T
        y, calls = torch.empty(t, rows + 3, dtype=torch.bfloat16, device="cuda"), []
        for _ in range(3):
            y.fill_(7.0)
            native_util.dense_stream(backend, packed, k, [dict(row0=0, rows=rows)], x, [(y, 0)])
            _close(y[:, :rows], want, 4e-3)
            assert bool((y[:, rows:] == 7).all())
            calls.append(y.clone())
        assert torch.equal(calls[0], calls[1]) and torch.equal(calls[0], calls[2])
        f = torch.ones(t, rows, device="cuda")
        native_util.dense_stream(backend, packed, k, [dict(row0=0, rows=rows, mul=0.5)], x, [(f, 2)])
        _close(f, 1 + 0.5 * want, 1e-5)


def test_segments(backend):
    import torch

    rows, ks, ins, acts = (300, 96, 1000, 64), (640, 640, 320, 64), (0, 0, 1, 1), (1, 0, 4, 2)
    k_pad, segs, blocks, outs, want = 640, [], [], [], []
    x, x2 = _bf16(6, 640, 1), _bf16(6, 384, 2)
    bias = torch.linspace(-1, 1, 300, device="cuda")
    row0 = 0
    for i, (r, k) in enumerate(zip(rows, ks)):
        pad = (r + 127) // 128 * 128
        w = torch.zeros(pad, k_pad, dtype=torch.bfloat16, device="cuda")
        w[:r, :k] = _bf16(r, k, 10 + i, k ** -0.5)
        blocks.append(w)
        segs.append(dict(row0=row0, rows=r, inp=ins[i], k=k, act=acts[i], bias=bias if i == 0 else None))
        row0 += pad
        z = (x2 if ins[i] else x)[:, :k].double() @ w[:r, :k].double().T + (bias.double() if i == 0 else 0.0)
        want.append({0: z, 1: z * z.sigmoid(), 2: z.sigmoid(), 4: z.clamp(min=0).square()}[acts[i]])
        outs.append((torch.empty(6, r, dtype=torch.float32, device="cuda"), 1))
    packed = native_util.dense_layout(torch.cat(blocks))
    for _ in range(2):
        for o, _ in outs:
            o.fill_(1e6)
        native_util.dense_stream(backend, packed, k_pad, segs, x, outs, x2=x2)
        for (o, _), z in zip(outs, want):
            _close(o, z, 1e-5)


def test_a_wait_that_gave_up_is_named(backend):
    """The code that the kernel leaves in the device error word, as the next host call reports it."""
    import ctypes as C

    f = backend.L._ZN5prism19device_error_resultEP14prism_cuda_ctxj
    f.restype, f.argtypes = C.c_int, [C.c_void_p, C.c_uint32]
    assert f(backend.ctx, 7) == -8  # PRISM_E_TIMEOUT
    assert b"streaming dense linear" in backend.L.prism_cuda_last_error(backend.ctx)
    backend.synchronize()
