"""A latent mixer, whose products go through the dense GEMM with k cut into ranges (split sums in scratch of the context), beside
a mixer of another kind on a stream of its own, on either side of the pair: against the restatement, and the same bits twice.

Tolerance: that of the other 16-bit runs."""
import numpy as np
import pytest

import layered_util as u
from oracle import layered as orc

pytestmark = pytest.mark.gpu
LATENT = u.latent(2, 64, 32, 64, 4096, 256, window=200)["mixer"]  # queries from 4096: 64 stages, few tiles
OTHERS = {"lightning": u.lightning(2, 64, 64)["mixer"], "attention": u.attention(4, 2, 32, 32, window=90), "gated_delta": u.delta(2, 2, 32, 32)}


@pytest.fixture
def any_pair(monkeypatch):
    """Layer type "any_pair": mixers of any two kinds."""
    from prism_engine_b200 import models as m

    def spec(x):
        return m.LayerSpec(**m.MIXERS[x["kind"]](x["mixer"]))

    def restated(h, w, mx, eps):
        sides = [orc.rms_norm(orc.MIXERS[mx[s]["kind"]](h, orc._sub(w, s + "."), mx[s]["mixer"], eps), w[s + ".out"], eps) for s in ("left", "right")]
        return 0.5 * (sides[0] + sides[1])

    monkeypatch.setitem(m.MIXERS, "any_pair", lambda x: dict(mixer=m.MIXER_PAIR, left=spec(x["left"]), right=spec(x["right"])))
    monkeypatch.setitem(orc.MIXERS, "any_pair", restated)


@pytest.mark.parametrize("latent_left", [True, False])
@pytest.mark.parametrize("kind", sorted(OTHERS))
def test_latent_beside_another(backend, any_pair, kind, latent_left):
    two = [{"kind": "latent_attention", "mixer": LATENT}, {"kind": kind, "mixer": OTHERS[kind]}]
    layer = {"type": "any_pair", "mixer": dict(zip(("left", "right"), two if latent_left else two[::-1])), "mlp": {"kind": "dense", "ff": 256}}
    cfg = u.sequential([layer, layer], width=128, vocab=128)
    w = u.sequential_weights(cfg, seed=3)
    toks = np.random.default_rng(4).integers(0, 128, 300).astype(np.uint32)
    want = u.expected(cfg, w, toks, "bfloat16")
    eng = u.engine(backend, cfg, w, dtype="bfloat16", max_seq=300)
    runs = []
    for _ in range(3):
        seq = eng.open_sequence()
        runs.append(eng.extend([(seq, toks, list(range(300)))]))
        eng.close_sequence(seq)
        assert u.error(runs[-1], want) <= u.TOL["bfloat16"]
    assert np.array_equal(runs[0], runs[1]) and np.array_equal(runs[0], runs[2])
    eng.close()
