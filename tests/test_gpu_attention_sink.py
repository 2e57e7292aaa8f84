"""The decode-attention kernel where one key takes nearly all the weight and its value row is zero (a first token that all
heads attend to): the output is the sum of small weights.  Against the same attention in 64 bits on the rotated query.

Tolerance: the rounding of the fp16 output (at most 2^-11 of a value, 2.8e-4 in the mean) is far above scores, sums and parts
of weights, of which the parts resolve 2^-38 of the largest weight, 2^-12 of a weight at e^-18 at most and a quarter of that
in the mean: 4e-4 of the norm."""
import numpy as np
import pytest

from prism_engine_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lead", [4.0, 10.0, 14.0, 18.0])
@pytest.mark.parametrize("hd,nh,nkv", [(32, 5, 1), (64, 14, 2), (128, 9, 1), (256, 3, 1)])
def test_small_weights_beside_a_large_one(backend, oracle, hd, nh, nkv, lead):
    n, kvd, c = 700, nkv * hd, hd // 2 - 1  # element c turns slowly
    as_f = lambda b: b.view(np.float16).astype(np.float64)  # noqa: E731
    bits = lambda a: np.ascontiguousarray(a, np.float16).view(np.uint16)  # noqa: E731
    q = as_f(synth.make_activation(nh * hd, seed=3)).reshape(nh, hd) * 0.5
    K, V = as_f(synth.make_activation((n, kvd), seed=1)).reshape(n, nkv, hd), as_f(synth.make_activation((n, kvd), seed=2)) * 8192.0
    q[:, c], q[:, c + hd // 2], K[:, :, c], K[:, :, c + hd // 2] = 4.0, 0.0, 0.0, 0.0
    K[0], V[0] = 0.0, 0.0
    K[0, :, c] = lead / 4.0 * hd ** 0.5
    q, K, V = bits(q).reshape(-1), bits(K).reshape(n, kvd), bits(V)
    turned = as_f(oracle.rope(q, n - 1, hd, 1e4)).reshape(nh, hd)
    k, v = as_f(K).reshape(n, nkv, hd), as_f(V).reshape(n, nkv, hd)
    want = np.empty((nh, hd))
    for h in range(nh):
        s = k[:, h // (nh // nkv)] @ turned[h] / np.sqrt(hd)
        w = np.exp(s - s.max())
        want[h] = (w / w.sum()) @ v[:, h // (nh // nkv)]
    backend.kv_init(1, kvd, 1024)
    for p in range(n - 1):
        backend.append_kv(0, K[p], V[p], p)
    for cluster in (0, 1):
        backend.set_option("attn_cluster", cluster)
        try:
            got = backend.attention_step_kv(0, q, K[-1], V[-1], n - 1, nh, nkv, hd, rope_k=False, rope_base=1e4)
        finally:
            backend.set_option("attn_cluster", 0)
        err = np.linalg.norm(as_f(got) - want.reshape(-1)) / np.linalg.norm(want)
        assert err <= 4e-4, (cluster, err)
