"""Device memory that the quantiser's host call leaves with the context: nothing of a large matrix, at most 64 MB of smaller ones, and
that only until something else of the context needs it."""
import numpy as np
import pytest

import prism_engine_b200 as p

pytestmark = pytest.mark.gpu


def _free():
    import torch

    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def test_what_stays_with_the_context():
    with p.CudaBackend(device=0) as be:
        small = np.zeros((512, 512), np.float32)
        be.palettize(small)  # kernels loaded
        be.palettize(np.zeros((8192, 512), np.float32))
        before = _free()
        be.palettize(np.zeros((16384, 2048), np.float32))  # 128 MB
        assert _free() >= before - (4 << 20)
        be.palettize(np.zeros((3584, 3584), np.float32))
        assert before - (64 << 20) <= _free() <= before + (64 << 20)
        assert _free() < before  # kept for the next of its size


@pytest.mark.parametrize("what", ["cache", "weights"])
def test_another_allocation_takes_it_back(what):
    import torch

    with p.CudaBackend(device=0) as be:
        be.synth("s", 64, 128)  # kernels loaded
        be.palettize(np.zeros((3584, 3584), np.float32))
        kept = 3584 * 3584 * 4 + 3584 * 3584 // 2
        hog = torch.empty(_free() - (160 << 20), dtype=torch.uint8, device="cuda")
        try:
            if what == "cache":
                kv_dim, rows = 1024, (_free() + kept // 2) // (2 * 2 * 1024)
                be.kv_init(1, kv_dim, rows)
            else:
                rows = (_free() + kept // 2) * 2 // 4096
                be.synth("w", rows, 4096)
        finally:
            del hog
            torch.cuda.empty_cache()
