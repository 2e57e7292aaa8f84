"""Prompts of several sequences in one portion against the same prompts in calls of their own: spans of one row and of many, prompts that
portions cut, sequences that are not at their beginning.

Tolerance: the linears see other row counts (other kernels below nine rows, other orders of sums): bf16 activations differ by roundings,
2^-8 each, that travel through two layers, 2e-2 of the norm as for the oracle; fp32 sums 1e-5."""
import numpy as np
import pytest

import layered_util as lu

pytestmark = pytest.mark.gpu
MODELS = {
    "lightning_latent": lambda: lu.model([lu.lightning(2, 16, 24, ff=88), lu.latent(3, 16, 8, 16, 24, 48, window=24, ff=40)]),
    "pair_moe": lambda: lu.tozarax([lu.pair(lu.attention(4, 2, 8, 16, window=12), lu.delta(2, 1, 16, 24), lu.moe(4, 4, 24))] * 2),
}


@pytest.mark.parametrize("dtype,tol", [("bfloat16", 2e-2), ("float32", 1e-5)])
@pytest.mark.parametrize("name", sorted(MODELS))
@pytest.mark.parametrize("chunk", [2048, 32])
def test_together_as_apart(name, dtype, tol, chunk):
    import prism_engine_b200 as p

    raw = MODELS[name]()
    cfg = p.LayeredConfig.from_dict(raw)
    rng = np.random.default_rng(3)
    w = {}
    for tensor, shape in cfg.tensor_shapes().items():
        v = rng.normal(0.0, 1.0 / np.sqrt(shape[-1]) if len(shape) == 2 else 0.2, shape) + (len(shape) == 1 and not tensor.endswith(".b"))
        w[tensor] = (v.astype(np.float32).view(np.uint32) >> 16).astype(np.uint16)
    lens = [(40, 33), (2, 9), (9, 2), (33, 1), (5, 70)]
    prompts = [[rng.integers(0, raw["vocab"], n).tolist() for n in pair] for pair in lens]

    def logits(together):
        with p.CudaBackend(device=0) as be:
            be.set_option("layered_chunk", chunk)
            eng = p.PrismEngine(be, cfg, dtype=dtype, max_seq=128, max_batch=8)
            for tensor, v in w.items():
                eng.set_tensor(tensor, v)
            seqs, out = [eng.open_sequence() for _ in lens], []
            for turn in range(2):
                entries = [(q, pr[turn], sorted({0, len(pr[turn]) - 1})) for q, pr in zip(seqs, prompts)]
                out += [eng.extend(entries)] if together else [eng.extend([entry]) for entry in entries]
            eng.close()
            return np.concatenate(out)

    got, want = logits(True), logits(False)
    assert got.shape == want.shape
    assert np.linalg.norm(got - want) <= tol * np.linalg.norm(want)
