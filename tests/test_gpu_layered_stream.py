"""Layered models whose linears are large enough for the streaming kernel (2^24 weights; 2^25 where a norm is split off for it), both
arrangements: captured steps of 1, 2, 3 and 8 rows with prompts between them, whose split GEMMs use the same partial sums and arrival
counters, against the path without it (option fuse 0: a norm, then the tensor-core GEMM).

Tolerance: bf16 activations, other orders of fp32 sums, two layers: 2e-2 of the norm as for the oracle."""
import numpy as np
import pytest

import layered_util as lu

pytestmark = pytest.mark.gpu
MODELS = {
    # norm, in | lightning | norm and gate, out: the in, out and head linears have 2^26, 1.25 x 2^25 and 2^25 weights
    "parallel": (lambda: lu.model([lu.lightning(16, 128, 128, ff=8192)] * 2, width=4096, vocab=8200), 1 + 2 * 5 + 2 + 2),
    # in, the pair's out (two inputs, 2^24), in2 and down stream; the head (2^24, its norm folded in) does not
    "sequential": (lambda: lu.tozarax([lu.pair(lu.attention(16, 4, 128, 128), lu.delta(16, 16, 128, 128), {"kind": "dense", "ff": 8192})] * 2,
                                      width=4096, vocab=4104), None),
}


@pytest.mark.parametrize("name", sorted(MODELS))
def test_steps_and_prompts(name):
    import prism_engine_b200 as p

    raw, kernels = MODELS[name][0](), MODELS[name][1]
    cfg = p.LayeredConfig.from_dict(raw)

    def logits(fuse):
        rng = np.random.default_rng(4)
        tokens = lambda n: rng.integers(0, raw["vocab"], n).tolist()  # noqa: E731
        with p.CudaBackend(device=0) as be:
            be.set_option("fuse", fuse)
            eng = p.PrismEngine(be, cfg, dtype="bfloat16", max_seq=256, max_batch=8)
            eng.synth_weights(seed=5, sigma=0.02)
            seqs, out, counts = [eng.open_sequence() for _ in range(8)], [], []
            out.append(eng.extend([(q, tokens(9 + i), [0, 8]) for i, q in enumerate(seqs)]))
            for rows in (1, 2, 3, 8, 1):
                for _ in range(3):  # eager, captured, replayed
                    out.append(eng.extend([(q, tokens(1), [0]) for q in seqs[:rows]]))
                counts.append(eng.kernels_per_step())
                out.append(eng.extend([(seqs[7], tokens(33), [32])]))
            eng.close()
        return out, counts

    got, counts = logits(1)
    want, _ = logits(0)
    if kernels:
        assert counts[0] == counts[-1] == kernels, counts
    for i, (a, b) in enumerate(zip(got, want)):
        assert a.shape == b.shape and np.linalg.norm(a - b) <= 2e-2 * np.linalg.norm(b), (i, np.linalg.norm(a - b) / np.linalg.norm(b))
