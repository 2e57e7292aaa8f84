"""Options of which "the engine's choice" is the default: a caller who set one can return to it.  Seen in the number of
kernels that a call launches and in the last bits of the logits (another kernel adds in another order).  Where an option names
kernels, those run and not the register-palette kernel."""
import numpy as np
import pytest

import native_util
import prism_engine_b200 as p
from prism_engine_b200 import synth

pytestmark = pytest.mark.gpu
CFG = dict(num_layers=1, hidden_size=1024, num_heads=8, num_kv_heads=2, head_dim=128, intermediate_size=16384, vocab_size=512,
           norm_eps=1e-6, rope_theta=1e6, tie_word_embeddings=False)


def test_the_engines_choice_can_be_set_again():
    with p.CudaBackend(device=0) as be:
        eng = p.PrismEngine(be, p.model_config(**CFG, max_seq=900, max_batch=8, profile="baseline"))
        eng.synth_weights(seed=1)
        prompts = np.stack([synth.make_prompt(40, 512, seed=s) for s in range(8)])

        def trace():
            eng.reset(8)
            before = be.launch_count()
            _, logits = eng.step(np.arange(8, dtype=np.uint32) + 3, want_logits=True)
            step = be.launch_count() - before
            before = be.launch_count()
            eng.generate(prompts, 1)
            return step, logits.tobytes(), be.launch_count() - before

        for option, own, other in (("batch_gemv_max", 0, 8), ("prefill_chunk", -1, 16)):
            trace()  # scratch has grown
            be.set_option(option, own)
            first = trace()
            be.set_option(option, other)
            changed = trace()
            be.set_option(option, own)
            assert trace() == first and changed != first, option
            with pytest.raises(p.PrismCudaError):
                be.set_option(option, own - 1)
        eng.close()


@pytest.mark.parametrize("option,own,others", [("batch_gemv_max", 0, (1, 8, 64)), ("gemv_variant", 1, (0, 2, 3, 4, 5)), ("gemm_variant", 1, (0,))])
@pytest.mark.parametrize("bits,tokens", [(2, 2), (2, 7), (2, 8), (4, 3), (4, 16), (2, 32)])
def test_a_caller_who_names_the_kernels_gets_them(bits, tokens, option, own, others):
    import torch

    m, k = 896, 4864
    with p.CudaBackend(device=0) as be:
        h = be.upload("w", synth.make_payload(m, k, bits=bits, seed=1), m, k, bits)
        x, y = torch.randn(tokens, k, device="cuda").half(), torch.empty(tokens, m, dtype=torch.float16, device="cuda")
        assert native_util.few_tokens_taken(be, h, x, y)
        for other in others:
            be.set_option(option, other)
            assert not native_util.few_tokens_taken(be, h, x, y), other
        be.set_option(option, own)
        assert native_util.few_tokens_taken(be, h, x, y)
