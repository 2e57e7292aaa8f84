"""The dense GEMM on pairs of CTAs, with its k cut into ranges: few row tiles and a long k (a model whose feed-forward is
much wider than the model), token counts at the edges of the 64 / 128 / 256-token tiles, against the float64 restatement.

Tolerance: the one of the other 16-bit runs (activations rounded to bf16 between the linears); and the same input twice
gives the same bits, whichever split of k arrives last."""
import numpy as np
import pytest

import layered_util as u
from oracle import layered as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width,ff", [(256, 4096), (384, 6144)])
def test_few_rows_and_a_long_k(backend, width, ff):
    cfg = u.model([u.lightning(2, 64, 64, ff=ff)], width=width, vocab=256)
    w = u.weights(cfg, seed=ff)
    eng = u.engine(backend, cfg, w, dtype="bfloat16", max_seq=600)
    toks = np.random.default_rng(1).integers(0, 256, 520).astype(np.uint32)
    want = orc.forward(cfg, w, toks)
    for n in (9, 16, 63, 64, 65, 128, 129, 257, 520):
        seq = eng.open_sequence()
        got = eng.extend([(seq, toks[:n], list(range(n)))])
        eng.close_sequence(seq)
        assert u.error(got, want[:n]) <= u.TOL["bfloat16"], n
        seq = eng.open_sequence()
        again = eng.extend([(seq, toks[:n], list(range(n)))])
        eng.close_sequence(seq)
        assert np.array_equal(got, again), n
    eng.close()


def test_a_longer_prompt_after_the_step_was_captured(backend):
    """Scratch that a captured step uses grows with a later, longer portion: the step is captured again."""
    cfg = u.model([u.lightning(2, 64, 64, ff=4096)], width=256, vocab=256)
    w = u.weights(cfg, seed=5)
    eng = u.engine(backend, cfg, w, dtype="bfloat16", max_seq=600, max_batch=12)
    toks = np.random.default_rng(2).integers(0, 256, 500).astype(np.uint32)
    want = orc.forward(cfg, w, toks[:16])
    for longer in (20, 500):
        seqs = [eng.open_sequence() for _ in range(12)]
        got = [eng.extend([(s, toks[t:t + 1], [0]) for s in seqs]) for t in range(8)]  # eager, captured, replayed
        for t in range(8):
            assert u.error(got[t], np.repeat(want[t:t + 1], 12, 0)) <= u.TOL["bfloat16"]
        for s in seqs:
            eng.close_sequence(s)
        s = eng.open_sequence()
        eng.extend([(s, toks[:longer], [longer - 1])])
        eng.close_sequence(s)
    eng.close()
