"""gemm_dev with Y over X, whole or in part: bit for bit what it gives into memory of its own."""
import numpy as np
import pytest

from prism_engine_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,k", [(512, 512), (256, 512), (1024, 384), (1032, 96)])
def test_y_over_x(backend, m, k):
    import torch

    h = backend.upload("in_place", synth.make_payload(m, k, seed=m + k), m, k)
    try:
        for t in (1, 7, 8, 33, 300, 1030):
            x = torch.from_numpy(np.random.default_rng(t).standard_normal((t, k)).astype(np.float16)).cuda()
            want = torch.empty(t, m, dtype=torch.float16, device="cuda")
            torch.cuda.synchronize()
            backend.gemm_dev(h, x.data_ptr(), t, want.data_ptr())
            for off in (0, 8 * (t * min(m, k) // 16), -8 * (t * min(m, k) // 16)):  # halfs from X's start to Y's
                buf = torch.zeros(t * (2 * k + 2 * m), dtype=torch.float16, device="cuda")
                x0 = max(0, -off)
                buf[x0:x0 + t * k] = x.reshape(-1)
                torch.cuda.synchronize()
                backend.gemm_dev(h, buf[x0:].data_ptr(), t, buf[x0 + off:].data_ptr())
                backend.synchronize()
                assert torch.equal(buf[x0 + off:x0 + off + t * m].view(t, m), want), (t, off)
    finally:
        backend.free(h)
