"""Row buffers of a layered model: a portion of several short sequences takes at most an eighth of the memory that is left, else it
shrinks; more sequences add caches, and rows only up to 2048 however many tokens one sequence may have at once.

The logits of a smaller portion differ as in test_gpu_layered_portions.py: other row counts, bf16 roundings, 2e-2 of the norm."""
import numpy as np
import pytest

import layered_util as lu

pytestmark = pytest.mark.gpu
WIDTH, LAYERS, SEQS, MAX_SEQ = 1024, 8, 24, 96


def _model(chunk=2048, max_seq=MAX_SEQ, max_batch=SEQS, layers=LAYERS, hog_to=None, run=True):
    """Bytes that creating the model takes, and logits of prompts in one call; hog_to: bytes of the GPU that are free before."""
    import torch

    import prism_engine_b200 as p

    cfg = p.LayeredConfig.from_dict(lu.tozarax([lu.pair(lu.attention(8, 2, 128, 128), lu.delta(8, 8, 128, 128), lu.moe(4, 4, 64))] * layers, width=WIDTH, max_positions=4096))
    hog = None
    with p.CudaBackend(device=0) as be:
        be.set_option("layered_chunk", chunk)
        torch.cuda.synchronize()
        if hog_to:
            hog = torch.empty(torch.cuda.mem_get_info()[0] - hog_to, dtype=torch.uint8, device="cuda")
        before = torch.cuda.mem_get_info()[0]
        eng = p.PrismEngine(be, cfg, dtype="bfloat16", max_seq=max_seq, max_batch=max_batch)
        kept = before - torch.cuda.mem_get_info()[0]
        logits = None
        if run:
            eng.synth_weights(seed=3, sigma=0.02)
            rng = np.random.default_rng(0)
            entries = [(eng.open_sequence(), rng.integers(0, 131, MAX_SEQ - 3 - i % 5).tolist(), [0, 50]) for i in range(SEQS)]
            logits = eng.extend(entries)
        eng.close()
    del hog
    torch.cuda.empty_cache()
    return kept, logits


def test_portions_shrink_when_memory_is_short():
    _model()  # kernels loaded
    plenty, want = _model()
    history = (LAYERS + 1) * WIDTH * 4
    short, got = _model(hog_to=1200 << 20)
    assert plenty - short >= 1000 * history, (plenty >> 20, short >> 20)
    assert np.linalg.norm(got - want) <= 2e-2 * np.linalg.norm(want)


def test_sequences_beside_add_caches_and_no_rows():
    _model(layers=1)
    one, _ = _model(chunk=65536, max_seq=4096, max_batch=1, layers=1, run=False)
    many, _ = _model(chunk=65536, max_seq=4096, max_batch=16, layers=1, run=False)
    kept_by_a_sequence = 4096 * 2 * 8 * 128 * 2 + 8 * 128 * 128 * 4 + (1 << 20)  # keys and values, state, rings of convolutions
    assert many - one <= 15 * kept_by_a_sequence + (16 << 20), (one >> 20, many >> 20)
