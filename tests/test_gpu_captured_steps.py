"""When a decode step is captured: the first one runs eagerly and grows what scratch it needs, the second is captured, and
host calls that only grow staging buffers leave the captured step alone.  Counted in kernel launches (a replay is one)."""
import numpy as np
import pytest

import layered_util as u
import prism_engine_b200 as p

pytestmark = pytest.mark.gpu
CFG = dict(num_layers=2, hidden_size=1024, num_heads=8, num_kv_heads=2, head_dim=128, intermediate_size=4096, vocab_size=2048,
           norm_eps=1e-6, rope_theta=1e6, tie_word_embeddings=False)


def _launches(be, step, n):
    out = []
    for i in range(n):
        before = be.launch_count()
        step(i)
        out.append(be.launch_count() - before)
    return out


@pytest.mark.parametrize("batch", [1, 4, 12])
def test_second_step_is_captured(batch):
    with p.CudaBackend(device=0) as be:
        eng = p.PrismEngine(be, p.model_config(**CFG, max_seq=32, max_batch=batch, profile="baseline"))
        eng.synth_weights(seed=1)
        eng.reset(batch)
        n = _launches(be, lambda i: eng.step(np.full(batch, 3 + i, np.uint32)), 4)
        assert n[0] > 10 and n[1] == n[2] == n[3] < n[0], n
        be.vec_add(np.zeros(1 << 22, np.uint16), np.zeros(1 << 22, np.uint16))  # staging grows past anything before it
        assert _launches(be, lambda i: eng.step(np.full(batch, 9, np.uint32)), 1) == [n[3]]
        eng.close()


@pytest.mark.parametrize("batch", [1, 12])
def test_second_layered_step_is_captured(batch):
    cfg = u.model([u.lightning(2, 64, 64, ff=4096)], width=256, vocab=256)
    with p.CudaBackend(device=0) as be:
        eng = u.engine(be, cfg, u.weights(cfg, seed=1), dtype="bfloat16", max_seq=64, max_batch=batch)
        seqs = [eng.open_sequence() for _ in range(batch)]
        n = _launches(be, lambda i: eng.extend([(s, np.array([5 + i], np.uint32), [0]) for s in seqs]), 4)
        assert n[1] == n[2] == n[3] < n[0], n
        eng.close()


def test_logits_of_the_rows_that_want_them(backend):
    """Steps of several rows of which some want logits, once or twice, alone or side by side, and a step whose logits are more
    than the model's pinned memory: what each row gets is what it gets alone with all rows wanting."""
    for vocab in (256, 900000):
        cfg = u.model([u.lightning(2, 64, 64, ff=128)], width=128, vocab=vocab)
        eng = u.engine(backend, cfg, u.weights(cfg, seed=1), dtype="bfloat16", max_seq=16, max_batch=6)
        tokens = [np.array([7 + 3 * i], np.uint32) for i in range(6)]

        def step(wants):
            seqs = [eng.open_sequence() for _ in range(6)]
            out = eng.extend([(s, t, w) for s, t, w in zip(seqs, tokens, wants)])
            for s in seqs:
                eng.close_sequence(s)
            return out

        alone = [step([[0] if i == j else [] for i in range(6)])[0] for j in range(6)]
        assert not np.array_equal(alone[0], alone[1])
        for wants in ([1, 1, 1, 1, 1, 1], [0, 1, 2, 0, 0, 1], [0, 0, 0, 0, 2, 1], [0, 0, 0, 0, 0, 0]):
            got = step([[0] * n for n in wants])
            rows = [j for j, n in enumerate(wants) for _ in range(n)]
            assert len(got) == len(rows)
            for g, j in zip(got, rows):
                assert np.array_equal(g, alone[j]), (vocab, wants, j)
        eng.close()
