"""The decode-attention kernel with infinities and NaN among cached and new rows, against the oracle's rope_inplace +
attention_cpu: the same outputs are infinite (of the same sign) and NaN, the others agree.

A weight of two 16-bit parts times an infinite value is NaN where a part is 0 or negative, and a tile of which every score
is -inf has no maximum to subtract; neither may show.  Tolerance of the finite outputs as in test_gpu_attention.py."""
import numpy as np
import pytest

from conftest import rel_l2
from prism_engine_b200 import synth

pytestmark = pytest.mark.gpu
HEADS = [(32, 5, 1), (64, 14, 2), (128, 9, 1), (256, 3, 1)]


def _rows(hd, nh, nkv, ctx_len):
    as_h = lambda b: b.view(np.float16).copy()  # noqa: E731
    kvd = nkv * hd
    return (as_h(synth.make_activation(nh * hd, seed=3)), as_h(synth.make_activation((ctx_len, kvd), seed=1)),
            as_h(synth.make_activation((ctx_len, kvd), seed=2)))


def _check(backend, oracle, hd, nh, nkv, q, K, V, cluster):
    ctx_len, pos = K.shape[0], K.shape[0] - 1
    bits = lambda a: np.ascontiguousarray(a).view(np.uint16)  # noqa: E731
    backend.set_option("attn_cluster", cluster)
    try:
        backend.kv_init(1, nkv * hd, 512)
        for p in range(pos):
            backend.append_kv(0, bits(K[p]), bits(V[p]), p)
        got = backend.attention_step_kv(0, bits(q), bits(K[pos]), bits(V[pos]), pos, nh, nkv, hd, rope_k=False, rope_base=1e4)
    finally:
        backend.set_option("attn_cluster", 0)
    want = oracle.attention(oracle.rope(bits(q), pos, hd, 1e4), bits(K).reshape(-1), bits(V).reshape(-1), nh, nkv, hd, ctx_len)
    g, w = (np.asarray(x, np.uint16).view(np.float16).astype(np.float64) for x in (got, want))
    assert np.array_equal(np.isnan(g), np.isnan(w))
    assert np.array_equal(np.where(np.isinf(g), g, 0), np.where(np.isinf(w), w, 0))
    finite = np.isfinite(w)
    if finite.any():
        assert rel_l2(got[finite], want[finite]) <= 1e-3
    return w


@pytest.mark.parametrize("cluster", [1, 8])
@pytest.mark.parametrize("hd,nh,nkv", HEADS)
def test_infinite_values(backend, oracle, hd, nh, nkv, cluster):
    """Some columns of some value rows, old and new, the signs meeting in one column."""
    for ctx_len in (2, 17, 300):
        q, K, V = _rows(hd, nh, nkv, ctx_len)
        V[0, 3], V[ctx_len // 2, 7], V[-1, 9] = np.inf, -np.inf, np.inf
        V[0, 11], V[-1, 11] = np.inf, -np.inf
        w = _check(backend, oracle, hd, nh, nkv, q, K, V, cluster)
        assert np.isinf(w).any() and np.isnan(w).any() and np.isfinite(w).any()


@pytest.mark.parametrize("cluster", [1, 8])
@pytest.mark.parametrize("hd,nh,nkv", HEADS)
def test_scores_of_minus_infinity(backend, oracle, hd, nh, nkv, cluster):
    """A whole tile of 16 positions that no head attends to, and single ones elsewhere."""
    ctx_len = 300
    q, K, V = _rows(hd, nh, nkv, ctx_len)
    bits = np.ascontiguousarray(q).view(np.uint16)
    q.reshape(nh, hd)[:, hd // 2 - 1] = 2.0  # turns slowly: positive in every head at any position of the test
    q.reshape(nh, hd)[:, hd - 1] = 0.0
    bits = np.ascontiguousarray(q).view(np.uint16)
    turned = oracle.rope(bits, ctx_len - 1, hd, 1e4).view(np.float16).reshape(nh, hd)
    assert (turned[:, hd // 2 - 1] > 0).all()
    for p in list(range(16, 32)) + [40, 299]:
        K[p].reshape(nkv, hd)[:, hd // 2 - 1] = -np.inf
    w = _check(backend, oracle, hd, nh, nkv, q, K, V, cluster)
    assert np.isfinite(w).all()


@pytest.mark.parametrize("hd,nh,nkv", HEADS)
def test_small_weight_of_an_infinite_value(backend, oracle, hd, nh, nkv):
    """A weight far below what 16 bits hold, on an infinite value: infinite, as in 32 bits."""
    q, K, V = _rows(hd, nh, nkv, 40)
    q[:], K[:] = 0.0, 0.0
    q.reshape(nh, hd)[:, hd // 2 - 1] = 8.0
    K[5].reshape(nkv, hd)[:, hd // 2 - 1] = 5.0 * hd ** 0.5  # about 40 above the others: weights of e^-40
    V[20, 2] = np.inf
    w = _check(backend, oracle, hd, nh, nkv, q, K, V, 0)
    assert np.isinf(w).any()


@pytest.mark.parametrize("what", ["q", "k", "v"])
def test_not_a_number(backend, oracle, what):
    for hd, nh, nkv in HEADS:
        q, K, V = _rows(hd, nh, nkv, 50)
        {"q": q, "k": K[20], "v": V[20]}[what][5] = np.nan
        w = _check(backend, oracle, hd, nh, nkv, q, K, V, 0)
        assert np.isnan(w).any()
