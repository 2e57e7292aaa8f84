"""The prompt-portion attention kernel by itself against the same attention in 64 bits, on the rotated queries and the cache
rows that it left.

Tolerance: scores and sums in fp32 and the weights' parts are far below the rounding of the fp16 outputs, at most 2^-11 of
a value, 2^-11 / sqrt(3) = 2.8e-4 in the mean: 4e-4 of the norm."""
import math

import pytest

import native_util

pytestmark = pytest.mark.gpu
HEADS = [(32, 6, 2), (64, 7, 1), (128, 4, 4), (256, 3, 1)]
TOL = 4e-4


def _inputs(nh, nkv, hd, tokens, seed=0):
    import torch

    g = torch.Generator(device="cuda").manual_seed(seed + hd)
    return torch.randn(tokens, (nh + 2 * nkv) * hd, device="cuda", generator=g).half()


def _attend(backend, qkv, nh, nkv, hd, T, page=0, **kw):
    """(kernel's output, 64-bit output), all tokens of one sequence in one portion behind `pos0` zero rows of cache."""
    import torch

    pos0, kvd = kw.pop("pos0", 0), nkv * hd
    n = pos0 + T
    rows, tbl = -(-n // (page or 1)) * (page or 1), None
    if page:
        tbl = torch.arange(rows // page, dtype=torch.int32, device="cuda").flip(0).reshape(1, -1).contiguous()
    kc, vc = (torch.zeros(rows, kvd, dtype=torch.float16, device="cuda") for _ in range(2))
    got = native_util.prompt_attention(backend, qkv, kc, vc, nh, nkv, hd, T, pos0=pos0, page_tbl=tbl, page=page, **kw).double()
    if page:
        kc, vc = (c.view(-1, page, kvd).flip(0).reshape(rows, kvd) for c in (kc, vc))
    q = qkv[:, :nh * hd].double().view(T, nh, hd)
    k, v = (c[:n].double().view(n, nkv, hd) for c in (kc, vc))
    seen = torch.arange(n, device="cuda")[None] <= pos0 + torch.arange(T, device="cuda")[:, None]
    want = torch.empty(T, nh, hd, dtype=torch.float64, device="cuda")
    for h in range(nh):
        s = (q[:, h] @ k[:, h // (nh // nkv)].T) / math.sqrt(hd)
        s = torch.where(seen, s, -math.inf)
        w = (s - s.nan_to_num(nan=-math.inf, neginf=-math.inf, posinf=math.inf).max(-1, keepdim=True).values).exp()
        w = torch.where(seen, w / w.sum(-1, keepdim=True), 0.0)
        vh = v[:, h // (nh // nkv)]
        bad = ~vh.isfinite()
        o = w @ vh.masked_fill(bad, 0.0)
        for p, d in bad.nonzero().tolist():  # what a sum over the seen positions alone makes of it
            o[max(0, p - pos0):, d] += w[max(0, p - pos0):, p] * vh[p, d]
        want[:, h] = o
    return got.view(T, nh, hd), want


def _compare(got, want):
    import torch

    limit = 65520.0  # rounds to an infinite fp16
    assert torch.equal(got.isnan(), want.isnan())
    assert torch.equal(torch.where(got.isinf(), got, 0.0), torch.where(want.abs() >= limit, want.sign() * math.inf, 0.0))
    ok = want.abs() < limit
    err = (got - want)[ok].norm() / want[ok].norm().clamp(min=1e-300)
    assert err <= TOL, float(err)


@pytest.mark.parametrize("page", [0, 16, 256])
@pytest.mark.parametrize("hd,nh,nkv", HEADS)
def test_infinite_values_stay_with_the_rows_that_see_them(backend, hd, nh, nkv, page):
    """Value rows that overflowed, in the first tile, at its end, alone in a last tile: rows before them are what they are without."""
    for T, at in ((300, (0, 127, 131, 299)), (129, (128,)), (2, (1,))):
        qkv = _inputs(nh, nkv, hd, T)
        v = qkv[:, (nh + nkv) * hd:]
        for i, p in enumerate(at):
            v[p, 3 + i] = math.inf if i % 2 else -math.inf
            v[p, 20] = -math.inf if i % 2 else math.inf
        got, want = _attend(backend, qkv, nh, nkv, hd, T, page=page)
        assert want.isinf().any() and want.isfinite().any()
        _compare(got, want)


@pytest.mark.parametrize("hd,nh,nkv", HEADS)
def test_keys_of_minus_infinity(backend, hd, nh, nkv):
    """A first tile in which later rows see nothing but scores of -inf, and single such keys."""
    import torch

    T = 300
    qkv = _inputs(nh, nkv, hd, T)
    c = hd // 2 - 1  # turns slowly
    qkv[:, :nh * hd].view(T, nh, hd)[:, :, c], qkv[:, :nh * hd].view(T, nh, hd)[:, :, c + hd // 2] = 2.0, 0.0
    k = qkv[:, nh * hd:(nh + nkv) * hd].view(T, nkv, hd)
    for p in list(range(1, 128)) + [200]:
        k[p, :, c] = -math.inf
    k[0, :, c] = -200.0 * hd ** 0.5  # weight 0 for every row that sees another key
    got, want = _attend(backend, qkv, nh, nkv, hd, T, rope_k=0)
    assert want.isfinite().all()
    _compare(got, want)
    k[0, :, c] = -math.inf  # rows of the first tile: no score at all
    got, want = _attend(backend, _inputs(nh, nkv, hd, T).copy_(qkv), nh, nkv, hd, T, rope_k=0)
    assert torch.equal(got.isnan(), want.isnan()) and want.isnan().any() and want.isfinite().any()


@pytest.mark.parametrize("what", ["q", "k", "v"])
def test_not_a_number(backend, what):
    for hd, nh, nkv in HEADS:
        T = 200
        qkv = _inputs(nh, nkv, hd, T)
        qkv[150, {"q": 0, "k": nh * hd, "v": (nh + nkv) * hd}[what] + 5] = math.nan
        got, want = _attend(backend, qkv, nh, nkv, hd, T)
        assert want.isnan().any() and want[:150].isfinite().all()
        _compare(got, want)


@pytest.mark.parametrize("hd,nh,nkv", HEADS)
def test_maximum_moves(backend, hd, nh, nkv):
    """Keys that grow along the prompt, scores of tens of nats: the maximum moves in every key tile, in some rows of a warp by
    more than the others, so sums and outputs of the tiles before are scaled down."""
    import torch

    T = 700
    qkv = _inputs(nh, nkv, hd, T)
    grow = (torch.arange(T, device="cuda")[:, None] / 64.0).exp2().clamp(max=30.0)
    qkv[:, nh * hd:(nh + nkv) * hd] = (qkv[:, nh * hd:(nh + nkv) * hd].float() * grow).half()
    _compare(*_attend(backend, qkv, nh, nkv, hd, T))


@pytest.mark.parametrize("lead", [4.0, 10.0, 13.0, 16.0])
@pytest.mark.parametrize("hd,nh,nkv", HEADS)
def test_one_key_takes_the_weight_and_carries_nothing(backend, hd, nh, nkv, lead):
    """The first position leads all scores by `lead` nats, its value row is zero: outputs are sums of weights of e^-lead.
    The parts of a weight resolve 2^-37 of the largest weight, a seventh of TOL of a weight of e^-16."""
    T = 700
    qkv = _inputs(nh, nkv, hd, T)
    c = hd // 2 - 1  # turns slowly
    q, k = qkv[:, :nh * hd].view(T, nh, hd), qkv[:, nh * hd:(nh + nkv) * hd].view(T, nkv, hd)
    q *= 0.25
    q[:, :, c], q[:, :, c + hd // 2] = 4.0, 0.0
    k[:, :, c], k[:, :, c + hd // 2] = 0.0, 0.0
    k[0] = 0.0
    k[0, :, c] = lead / 4.0 * hd ** 0.5
    v = qkv[:, (nh + nkv) * hd:]
    v *= 4096.0
    v[0] = 0.0
    got, want = _attend(backend, qkv, nh, nkv, hd, T, rope_k=0)
    _compare(got[1:], want[1:])
