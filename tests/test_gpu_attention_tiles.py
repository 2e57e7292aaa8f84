"""The decode-attention kernel where its tiles can go wrong, against the oracle's rope_inplace + attention_cpu: contexts at the
edges of 16 positions and of one tile per warp of a cluster, groups that leave heads of a tile unused or need a second one, a
cluster of 16 CTAs, scores far apart (the running maximum moves, weights underflow).

Tolerance as in test_gpu_attention.py: 1e-3 relative L2 of the fp16 output."""
import numpy as np
import pytest

from conftest import rel_l2
from prism_engine_b200 import synth

pytestmark = pytest.mark.gpu


def _run(backend, oracle, hd, nh, nkv, ctx_len, max_seq, scale=1.0, cluster=0):
    kvd, pos = nkv * hd, ctx_len - 1
    backend.set_option("attn_cluster", cluster)
    backend.kv_init(1, kvd, max_seq)
    as_f = lambda b: b.view(np.float16).astype(np.float32)  # noqa: E731
    K = (as_f(synth.make_activation((ctx_len, kvd), seed=ctx_len)) * scale).astype(np.float16).view(np.uint16)
    V = synth.make_activation((ctx_len, kvd), seed=ctx_len + 1)
    q = synth.make_activation(nh * hd, seed=ctx_len + 2)
    for p in range(pos):
        backend.append_kv(0, K[p], V[p], p)
    try:
        got = backend.attention_step_kv(0, q, K[pos], V[pos], pos, nh, nkv, hd, rope_k=False, rope_base=1e4)
    finally:
        backend.set_option("attn_cluster", 0)
    return got, oracle.attention(oracle.rope(q, pos, hd, 1e4), K.reshape(-1), V.reshape(-1), nh, nkv, hd, ctx_len)


@pytest.mark.parametrize("hd,nh,nkv", [(32, 5, 1), (64, 14, 2), (128, 9, 1), (256, 3, 1)])
def test_tile_edges(backend, oracle, hd, nh, nkv):
    for ctx_len in (1, 2, 15, 16, 17, 127, 128, 129, 300):
        for cluster in (0, 8):
            got, want = _run(backend, oracle, hd, nh, nkv, ctx_len, 512, cluster=cluster)
            assert rel_l2(got, want) <= 1e-3, (ctx_len, cluster)


@pytest.mark.parametrize("hd,nh,nkv", [(64, 7, 1), (128, 8, 1)])
def test_sixteen_ctas(backend, oracle, hd, nh, nkv):
    got, want = _run(backend, oracle, hd, nh, nkv, 4500, 5000)
    assert rel_l2(got, want) <= 1e-3


def test_scores_far_apart(backend, oracle):
    got, want = _run(backend, oracle, 64, 4, 1, 200, 512, scale=40.0)
    assert rel_l2(got, want) <= 1e-3
