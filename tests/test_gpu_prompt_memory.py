"""Device memory that a long prompt leaves with the engine: rows of 2048 tokens of the residual, its norm, q | k | v, the
attention and the activations, and at most 64 MB of partial sums."""
import numpy as np
import pytest

import prism_engine_b200 as p
from prism_engine_b200 import synth

pytestmark = pytest.mark.gpu


def test_rows_kept_for_a_portion():
    import torch

    h, inter = 1024, 16384
    with p.CudaBackend(device=0) as be:
        eng = p.PrismEngine(be, p.model_config(num_layers=1, hidden_size=h, num_heads=8, num_kv_heads=2, head_dim=128, intermediate_size=inter,
                                               vocab_size=512, norm_eps=1e-6, rope_theta=1e6, tie_word_embeddings=False, max_seq=2100, profile="baseline"))
        eng.synth_weights(seed=1)
        eng.generate(synth.make_prompt(8, 512, seed=1), 2)  # kernels loaded, step captured
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        eng.generate(synth.make_prompt(2048, 512, seed=1), 2)
        torch.cuda.synchronize()
        kept = before - torch.cuda.mem_get_info()[0]
        rows = 2048 * 2 * (2 * h + 12 * 128 + 8 * 128 + inter)
        assert kept <= rows + (64 << 20) + (16 << 20), (kept >> 20, rows >> 20)
        eng.close()
