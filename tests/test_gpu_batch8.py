"""Eight sequences in a decode step: the engine's choice against all linears through the tcgen05 GEMM (option batch_gemv_max 1) and through
the batched GEMV (8), three sets of kernels that add in other orders; gate and up on both sides of the lines of gemm_pays_at_8, for 4 bits
(10240 rows) and for 2 (2^25 weights together).  Tolerance as in test_gpu_prefill_attention.py: another order of the fp32 sums, one layer of fp16 roundings."""
import numpy as np
import pytest

import prism_engine_b200 as p
from conftest import rel_l2
from prism_engine_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bits", [4, 2])
@pytest.mark.parametrize("inter", [8192, 8160, 10240, 10112])
def test_choice_at_eight_sequences(inter, bits):
    cfg = dict(num_layers=1, hidden_size=2048, num_heads=16, num_kv_heads=2, head_dim=128, intermediate_size=inter, vocab_size=640,
               norm_eps=1e-6, rope_theta=1e6, tie_word_embeddings=False)
    prompts = np.stack([synth.make_prompt(9, cfg["vocab_size"], seed=s) for s in range(8)])

    def logits(most):
        with p.CudaBackend(device=0) as be:
            eng = p.PrismEngine(be, p.model_config(**cfg, max_seq=16, max_batch=8, bits=bits, profile="baseline"))
            eng.synth_weights(seed=2, sigma=0.02)
            if most:
                be.set_option("batch_gemv_max", most)
            return eng.generate(prompts, 3, return_logits=True)

    tokens, got = logits(0)
    arms = {most: logits(most) for most in (1, 8)}
    assert not np.array_equal(arms[1][1], arms[8][1]) and not np.array_equal(got, arms[8][1])  # other kernels
    for most, (other, want) in arms.items():
        for b in range(8):
            if np.array_equal(tokens[b], other[b]):
                assert rel_l2(got[b], want[b]) <= 3.2e-3, (most, b)
    assert np.mean(tokens == other) >= 0.9
