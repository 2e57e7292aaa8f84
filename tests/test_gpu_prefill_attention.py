"""The prompt-portion attention kernel (tcgen05) inside generate(), against the step-per-token path of the same engine
(the decode attention kernel, itself tested against the oracle) and, for the shortest, the oracle's tokens.

Prompt lengths sit at the edges of the 128-key and 128- / 256-query tiles, portions of 100 tokens start at positions that
are no multiple of either, and pages of 16 and 256 positions are smaller and larger than a key tile.

Tolerance: both paths round q, k, v and the output of every layer to fp16 (2^-11 relative) and keep the softmax in fp32;
the linears of the two paths add in another order.  Two layers of about ten such roundings: 1e-3 * sqrt(10) at most.
"""
import numpy as np
import pytest

import prism_engine_b200 as p
from conftest import rel_l2
from prism_engine_b200 import synth

pytestmark = pytest.mark.gpu
TOL = 3.2e-3


def _logits(be, eng, prompts, chunk):
    be.set_option("prefill_chunk", chunk)
    return eng.generate(prompts, 1, return_logits=True)


@pytest.mark.parametrize("page", [0, 16, 256])
@pytest.mark.parametrize("hd,nh,nkv", [(32, 6, 2), (64, 7, 1), (128, 4, 4), (256, 3, 1)])
def test_prompt_portions_match_the_step_path(hd, nh, nkv, page):
    cfg = dict(num_layers=2, hidden_size=256, num_heads=nh, num_kv_heads=nkv, head_dim=hd, intermediate_size=384, vocab_size=640,
               norm_eps=1e-6, rope_theta=1e6, tie_word_embeddings=False)
    with p.CudaBackend(device=0) as be:
        eng = p.PrismEngine(be, p.model_config(**cfg, max_seq=600, max_batch=2, profile="baseline", kv_page_size=page))
        eng.synth_weights(seed=hd + page, sigma=0.06)
        for n in (2, 127, 128, 129, 255, 257, 513):
            prompts = np.stack([synth.make_prompt(n, cfg["vocab_size"], seed=s) for s in range(2)])
            _, want = _logits(be, eng, prompts, 0)
            for chunk in (512, 100):
                _, got = _logits(be, eng, prompts, chunk)
                for b in range(2):
                    assert rel_l2(got[b], want[b]) <= TOL, (n, chunk, b, rel_l2(got[b], want[b]))


def test_stale_cache_rows_stay_out():
    """A shorter prompt after a longer one whose values overflowed: positions past its end hold infinities and NaN."""
    cfg = dict(num_layers=1, hidden_size=128, num_heads=2, num_kv_heads=1, head_dim=64, intermediate_size=256, vocab_size=512,
               norm_eps=1e-6, rope_theta=1e6, tie_word_embeddings=True)
    with p.CudaBackend(device=0) as be:
        eng = p.PrismEngine(be, p.model_config(**cfg, max_seq=300, profile="baseline"))
        eng.synth_weights(seed=1, sigma=0.06)
        short = synth.make_prompt(70, 512, seed=2)
        _, want = eng.generate(short, 1, return_logits=True)
        kept = be.find("model.layers.0.self_attn.v_proj.weight")
        huge = np.full(synth.payload_bytes(64, 128), 0, np.uint8)
        huge[:64 * 32] = np.full(64 * 16, 60000.0, np.float16).view(np.uint8)  # every weight 60000: the value rows overflow
        eng.bind("v", 0, be.upload("huge", huge, 64, 128))
        eng.generate(synth.make_prompt(250, 512, seed=3), 1)
        eng.bind("v", 0, kept)
        _, got = eng.generate(short, 1, return_logits=True)
        assert np.array_equal(got, want)
