"""Prompts of several sequences in one portion: generate() with the engine's own portion size and with ones that cut the
batch unevenly, against the step-per-token path of the same engine.  Sequence lengths are no multiple of the attention's
tiles, so tiles end inside the next sequence's rows.  Tolerance as in test_gpu_prefill_attention.py."""
import numpy as np
import pytest

import prism_engine_b200 as p
from conftest import rel_l2
from prism_engine_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("page", [0, 16])
@pytest.mark.parametrize("batch,n", [(2, 2), (5, 67), (3, 200), (2, 1500)])
def test_sequences_share_a_portion(batch, n, page):
    cfg = dict(num_layers=2, hidden_size=256, num_heads=4, num_kv_heads=2, head_dim=64, intermediate_size=384, vocab_size=640,
               norm_eps=1e-6, rope_theta=1e6, tie_word_embeddings=False)
    prompts = np.stack([synth.make_prompt(n, cfg["vocab_size"], seed=s) for s in range(batch)])

    def logits(chunk):
        with p.CudaBackend(device=0) as be:
            eng = p.PrismEngine(be, p.model_config(**cfg, max_seq=n + 2, max_batch=batch, profile="baseline", kv_page_size=page))
            eng.synth_weights(seed=3, sigma=0.06)
            if chunk is not None:
                be.set_option("prefill_chunk", chunk)
            return eng.generate(prompts, 1, return_logits=True)[1]

    want = logits(0)
    for chunk in (None, 150, 2 * n):
        got = logits(chunk)
        for b in range(batch):
            assert rel_l2(got[b], want[b]) <= 3.2e-3, (chunk, b)
