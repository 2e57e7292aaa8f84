"""Workloads of the framework, through its public entry points: what a user's program has it do.

Kinds of case:

* ``mlp``       one fused gate/up SwiGLU and down projection of one token on device buffers (``mlp_dev``);
* ``gemm``      one palettized linear over a portion of a prompt on device buffers (``gemm_dev``);
* ``generate``  a palettized Llama/Qwen2-family model: prompt and greedy decode (``PrismEngine.generate``);
* ``quantise``  the offline quantiser, fp32 matrix to palettized payload (``CudaBackend.palettize``);
* ``trace``     a model described layer by layer, as a trace replay drives it: prompts of several sequences in one
  step, then decode steps with given tokens (``open_sequence`` / ``extend`` / ``close_sequence``).

Widths are those of the framework's own model configurations (and generic odd ones in ``draw``); depth and vocabulary
of the large ones are cut so that a state fits beside others, with the layers : head ratio kept.  Palettized weights
have N(0, 1 / fan-in) palettes (variance of what ends in the residual divided by the number of sublayers, as models are
initialised) and uniform indices; the head's rows are the embedding's moved on by one (tied: the embedding itself), so
greedy choices have the margin they have in a trained model and do not hang on rounding.
"""
import math

import numpy as np
import torch

import prism_engine_b200 as prism

SHAPES = {
    # hidden, heads, kv_heads, head_dim, intermediate
    "0p5b": (896, 14, 2, 64, 4864),
    "7b": (3584, 28, 4, 128, 18944),
    "72b": (8192, 64, 8, 128, 29568),
}
THETA, EPS = 1e6, 1e-6


def listed():
    return [
        # the smallest call: one MLP of a sub-billion model for one token, launch and latency bound
        dict(name="mlp_0p5b", kind="mlp", hidden=896, inter=4864, bits=4),
        # the largest linear of a prompt: gate projection over 2048 tokens
        dict(name="gemm_7b_gate", kind="gemm", rows=18944, k=3584, tokens=2048, bits=4),
        # chat with a small model: whole 0.5B model, short prompt, one sequence
        _gen("decode_0p5b", "0p5b", layers=24, vocab=151936, tied=True, prompt=128, new=64),
        # the headline workload: single-sequence decode of the largest model
        _gen("decode_72b", "72b", layers=3, vocab=8064, prompt=512, new=32),
        # a small serving batch on the paged cache, prompts of an odd length
        _gen("decode_7b_batch8", "7b", layers=4, vocab=19008, batch=8, prompt=203, new=24, page=64),
        # a larger serving batch of short prompts
        _gen("decode_7b_batch32", "7b", layers=4, vocab=19008, batch=32, prompt=61, new=16),
        # the smaller weight format
        _gen("decode_7b_2bit", "7b", layers=4, vocab=19008, bits=2, prompt=77, new=32),
        # time to first token of an ordinary long prompt
        _gen("prefill_7b", "7b", layers=4, vocab=19008, prompt=2048, new=1),
        # a long document and a short answer
        _gen("long_7b", "7b", layers=2, vocab=9472, prompt=8190, new=8),
        # converting a checkpoint: one attention projection
        dict(name="quantise_7b_q", kind="quantise", rows=3584, cols=3584),
        # trace replay, lightning and latent attention layers
        _trace("trace_mefipel_7b", "mefipel", "7b", layers=4, vocab=19008, batch=4, prompt=509, steps=12),
        # trace replay, windowed attention beside a gated delta rule, with experts
        _trace("trace_tozarax_7b", "tozarax", "7b", layers=2, vocab=9472, batch=4, prompt=509, steps=12),
    ]


def _gen(name, shape, layers, vocab, prompt, new, batch=1, bits=4, tied=False, page=0):
    h, nh, nkv, hd, inter = SHAPES[shape]
    return dict(name=name, kind="generate", hidden=h, heads=nh, kv_heads=nkv, head_dim=hd, inter=inter, layers=layers, vocab=vocab,
                tied=tied, bits=bits, batch=batch, prompt=prompt, new=new, page=page)


def _trace(name, design, shape, layers, vocab, batch, prompt, steps, dtype="bfloat16"):
    h, nh, nkv, hd, inter = SHAPES[shape]
    return dict(name=name, kind="trace", design=design, hidden=h, heads=nh, kv_heads=nkv, head_dim=hd, inter=inter, layers=layers,
                vocab=vocab, batch=batch, prompt=prompt, steps=steps, dtype=dtype)


def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choices(["mlp", "gemm", "generate", "quantise", "trace"], [1, 2, 5, 1, 3])[0]
    bits = rng.choice([4, 4, 4, 2])
    if kind == "mlp":
        if rng.random() < 0.5:
            hidden, _, _, _, inter = SHAPES[rng.choice(sorted(SHAPES))]
            inter = inter // rng.choice([1, 2]) + 32 * rng.randint(0, 30)
        else:  # any multiple of what the index rows need
            hidden, inter = 16 * _log(rng, 8, 512), 16 * _log(rng, 16, 1024)
        return dict(kind=kind, hidden=hidden, inter=inter, bits=bits)
    if kind == "gemm":
        h, nh, nkv, hd, inter = SHAPES[rng.choice(["0p5b", "7b"])]
        rows, k = rng.choice([((nh + 2 * nkv) * hd, h), (h, nh * hd), (inter, h), (h, inter), (8 * _log(rng, 8, 1024), 128 * _log(rng, 1, 64))])
        return dict(kind=kind, rows=rows, k=k, tokens=_log(rng, 2, 2048), bits=bits)
    if kind == "quantise":
        return dict(kind=kind, rows=_log(rng, 16, 3584), cols=2 * _log(rng, 32, 1792))
    if kind == "generate":
        which = rng.choice(["0p5b", "7b", "72b", "odd"])
        if which == "odd":
            hd, nkv = rng.choice([32, 64, 128, 256]), rng.choice([1, 2, 3, 4])
            nh = nkv * rng.choice([1, 2, 5, 8])
            h, inter, most = 32 * _log(rng, 4, 64), 32 * _log(rng, 8, 160), 1024
        else:
            h, nh, nkv, hd, inter = SHAPES[which]
            most = 2048 if which == "72b" else 4096
        batch = 1 if rng.random() < 0.5 else _log(rng, 2, 40)
        return dict(kind=kind, hidden=h, heads=nh, kv_heads=nkv, head_dim=hd, inter=inter,
                    layers=rng.randint(2, 12) if which == "0p5b" else rng.randint(1, 2) if which == "72b" else rng.randint(1, 4),
                    vocab=8 * _log(rng, 125, 2400) + rng.choice([0, 0, 1, 5]), tied=rng.random() < 0.4, bits=bits, batch=batch,
                    prompt=_log(rng, 1, max(1, min(most, 2 * most // batch))), new=_log(rng, 1, 48), page=rng.choice([0, 0, 64]))
    design, small = rng.choice(["mefipel", "tozarax"]), rng.random() < 0.5
    dtype = "float32" if small and rng.random() < 0.25 else "bfloat16"
    batch = _log(rng, 1, 12)
    return _drop_name(_trace("", design, "0p5b" if small else "7b", layers=rng.randint(2, 4) if small else 2, vocab=8 * _log(rng, 125, 1184),
                             batch=batch, prompt=_log(rng, 2, 256 if dtype == "float32" else 2048 // batch), steps=_log(rng, 1, 24), dtype=dtype))


def _drop_name(case):
    case.pop("name")
    return case


# ---- inputs ------------------------------------------------------------------------------------------
def _rand(*key):
    g = torch.Generator(device="cuda")
    v = 0
    for k in key:
        v = (v * 1000003 + int(k) + 1) % (1 << 62)
    g.manual_seed(v)
    return g


def _palette_and_index(rows, k, bits, sigma, *key):
    g = _rand(rows, k, bits, *key)
    pal = torch.randn(rows, 1 << bits, device="cuda", generator=g).mul_(sigma)
    pal = (pal - pal.mean(1, keepdim=True)).sort(dim=1).values.half()  # weights of a row have no common offset
    idx = torch.randint(0, 256, (rows, k * bits // 8), device="cuda", generator=g, dtype=torch.uint8)
    return pal, idx


def _payload(pal, idx):
    return torch.cat([pal.view(torch.uint8).reshape(-1), idx.reshape(-1)]).cpu().numpy()


def _dense64(pal, idx):
    """Weights a palette and its packed indices stand for (lowest bits first), in 64 bits."""
    bits = {16: 4, 4: 2}[pal.shape[1]]
    out = torch.empty(idx.shape[0], idx.shape[1] * 8 // bits, dtype=torch.float64, device="cuda")
    for r in range(0, idx.shape[0], 4096):
        b, p = idx[r:r + 4096].long(), pal[r:r + 4096].double()
        parts = [(b >> s) & ((1 << bits) - 1) for s in range(0, 8, bits)]
        out[r:r + 4096] = p.gather(1, torch.stack(parts, dim=-1).reshape(b.shape[0], -1))
    return out


def _model_tensors(c, seed):
    """(role, layer) -> how to make its palettes and indices."""
    h, qd, kvd, inter = c["hidden"], c["heads"] * c["head_dim"], c["kv_heads"] * c["head_dim"], c["inter"]
    shapes = {"q": (qd, h), "k": (kvd, h), "v": (kvd, h), "o": (h, qd), "gate": (inter, h), "up": (inter, h), "down": (h, inter)}

    def make(role, layer):
        if role in shapes:
            m, k = shapes[role]
            sigma = k ** -0.5 if role not in ("o", "down") else (2 * c["layers"] * k) ** -0.5
            return _palette_and_index(m, k, c["bits"], sigma, seed, layer, sorted(shapes).index(role))
        pal, idx = _palette_and_index(c["vocab"], h, c["bits"], 1.0, seed, 1 << 20, 0)
        if role == "lm_head":
            return (pal.float() / 64).half().roll(1, 0), idx.roll(1, 0)
        return pal, idx

    names = [(r, layer) for layer in range(c["layers"]) for r in shapes] + [("embed", 0)] + ([] if c["tied"] else [("lm_head", 0)])
    return names, make


def _prompts(c, seed):
    return np.random.default_rng([seed, 77]).integers(0, c["vocab"], size=(c["batch"], c["prompt"]), dtype=np.uint32)


def _layered_raw(c):
    """config.json of a layered case."""
    h, nh, nkv, hd, inter = c["hidden"], c["heads"], c["kv_heads"], c["head_dim"], c["inter"]
    window = 1024 if h < 2048 else 2048
    raw = {"norm": {"eps": 1e-6}, "vocab": c["vocab"], "width": h}
    if c["design"] == "tozarax":
        left = dict(heads=nh, kv_heads=nkv, dim=hd, vdim=hd, scale=hd ** -0.5, mask={"size": window})
        right = dict(heads=nh, kv_heads=nh if h < 2048 else nh // 2, dim=hd, vdim=hd, conv=4)
        mlp = {"kind": "moe", "expert": {"ff": inter // 4}, "router": {"experts": 16, "top": 4, "groups": {"count": 4, "keep": 2}}}
        raw.update(architecture="Tozarax", canon={"taps": 4}, max_positions=4096,
                   layers=[{"type": "parallel", "mixer": {"left": left, "right": right}, "mlp": mlp}] * c["layers"])
        return raw
    decay = [1.0 - 2.0 ** (-4.0 - 6.0 * i / nh) for i in range(nh)]
    rot = dict(base=5e5, dims=hd // 2, scaling={"factor": 8.0, "fast": 16.0, "original": 4096, "slow": 2.0})
    q_rank, kv_rank = (448, 256) if h < 2048 else (1536, 512)
    mixers = [{"type": "lightning", "mixer": dict(heads=nh, dim=hd, vdim=hd, decay=decay)},
              {"type": "latent_attention", "mixer": dict(heads=nh, dim=hd, rot_dim=hd // 2, vdim=hd, q_rank=q_rank, kv_rank=kv_rank,
                                                         mask={"size": window}, scale=(hd + hd // 2) ** -0.5, rot=rot)}]
    raw.update(architecture="Mefipel", logit_scale=1.0, residual_mult=0.5,
               layers=[dict(mixers[i % 2], mlp={"kind": "dense", "ff": inter}) for i in range(c["layers"])])
    return raw


def _layered_weights(c, seed):
    """Name -> bf16 tensor.  Matrices N(0, 1 / fan-in); the experts of a layer have most of their weights in common, so a
    choice between two of nearly equal score does not hang on rounding."""
    shapes = prism.LayeredConfig.from_dict(_layered_raw(c)).tensor_shapes()
    offset, out, common = 1.0 if c["design"] == "tozarax" else 0.0, {}, {}
    for i, (name, shape) in enumerate(shapes.items()):
        g, leaf = _rand(seed, i, 5), name.split(".")[-1]
        v = torch.randn(shape, device="cuda", generator=g)
        if name == "final.norm" or leaf in ("norm1", "norm2"):
            v = 0.1 * v + 1.0 - offset
        elif leaf in ("norm", "out"):
            v = 0.1 * v + 1.0
        elif leaf == "dwa":
            v = 0.1 * v
            v[-1] += 1.0
        elif leaf == "A_log":
            v = (1.0 + 15.0 * torch.rand(shape, device="cuda", generator=g)).log()
        elif leaf == "dt_bias":
            v = 0.5 * v - 4.0
        elif leaf.startswith("canon") or leaf == "conv":
            v = 0.3 * v
        elif name == "pos":
            v = 0.2 * v
        elif len(shape) == 1:
            v = 0.1 * v
        elif name != "embed":
            v = v * shape[1] ** -0.5
        head, _, part = name.partition(".mlp.e")
        if part:
            common.setdefault((head, leaf), v)
            v = 0.995 * common[head, leaf] + 0.1 * v
        out[name] = v.to(torch.bfloat16)
    return out


def _trace_tokens(c, seed):
    """Per sequence its prompt (lengths differ) and the tokens of its decode steps."""
    r = np.random.default_rng([seed, 78])
    lens = [max(1, c["prompt"] - 7 * i % max(1, c["prompt"] // 2)) for i in range(c["batch"])]
    return [(r.integers(0, c["vocab"], size=n, dtype=np.uint32), r.integers(0, c["vocab"], size=c["steps"], dtype=np.uint32)) for n in lens]


def prepare(case, seed):
    c, be = case, prism.CudaBackend(device=0)
    s = {"kind": c["kind"], "be": be}
    if c["kind"] == "mlp":
        h, inter = c["hidden"], c["inter"]
        for i, (name, m, k) in enumerate((("gate", inter, h), ("up", inter, h), ("down", h, inter))):
            s[name] = be.upload(name, _payload(*_palette_and_index(m, k, c["bits"], k ** -0.5, seed, i)), m, k, c["bits"])
        s["x"] = torch.randn(h, device="cuda", generator=_rand(seed, 9)).half()
        s["y"] = torch.empty(h, device="cuda", dtype=torch.float16)
    elif c["kind"] == "gemm":
        s["w"] = be.upload("w", _payload(*_palette_and_index(c["rows"], c["k"], c["bits"], c["k"] ** -0.5, seed)), c["rows"], c["k"], c["bits"])
        s["x"] = torch.randn(c["tokens"], c["k"], device="cuda", generator=_rand(seed, 9)).half()
        s["y"] = torch.empty(c["tokens"], c["rows"], device="cuda", dtype=torch.float16)
    elif c["kind"] == "quantise":
        s["w"] = (torch.randn(c["rows"], c["cols"], device="cuda", generator=_rand(seed, 9)) * 0.02).cpu().numpy()
    elif c["kind"] == "generate":
        cfg = prism.model_config(c["layers"], c["hidden"], c["heads"], c["kv_heads"], c["head_dim"], c["inter"], c["vocab"], EPS, THETA,
                                 c["tied"], bits=c["bits"], max_seq=c["prompt"] + c["new"] + 1, max_batch=c["batch"], kv_page_size=c["page"])
        eng = s["eng"] = prism.PrismEngine(be, cfg)
        names, make = _model_tensors(c, seed)
        for role, layer in names:
            pal, idx = make(role, layer)
            eng.bind(role, layer, be.upload("%s.%d" % (role, layer), _payload(pal, idx), idx.shape[0], idx.shape[1] * 8 // c["bits"], c["bits"]))
        s["prompts"], s["new"] = _prompts(c, seed), c["new"]
    else:
        eng = s["eng"] = prism.PrismEngine(be, prism.LayeredConfig.from_dict(_layered_raw(c)), dtype=c["dtype"],
                                           max_seq=c["prompt"] + c["steps"] + 1, max_batch=c["batch"])
        for name, w in _layered_weights(c, seed).items():
            eng.set_tensor(name, w.view(torch.int16).cpu().numpy().view(np.uint16))
        s["tokens"], s["steps"] = _trace_tokens(c, seed), c["steps"]
    return s


# ---- one pass ----------------------------------------------------------------------------------------
def run(state):
    s, be = state, state["be"]
    if s["kind"] == "mlp":
        be.mlp_dev(s["gate"], s["up"], s["down"], s["x"].data_ptr(), s["y"].data_ptr())
        return s["y"]
    if s["kind"] == "gemm":
        be.gemm_dev(s["w"], s["x"].data_ptr(), s["x"].shape[0], s["y"].data_ptr())
        return s["y"]
    if s["kind"] == "quantise":
        return be.palettize(s["w"])
    eng = s["eng"]
    if s["kind"] == "generate":
        tokens, logits = eng.generate(s["prompts"], s["new"], return_logits=True)
        return {"tokens": tokens, "logits": logits.view(np.float16)}
    seqs = [eng.open_sequence() for _ in s["tokens"]]
    out = [eng.extend([(q, prompt, [len(prompt) - 1]) for q, (prompt, _) in zip(seqs, s["tokens"])])]
    for i in range(s["steps"]):
        out.append(eng.extend([(q, after[i:i + 1], [0]) for q, (_, after) in zip(seqs, s["tokens"])]))
    for q in seqs:
        eng.close_sequence(q)
    return np.concatenate(out)


# ---- what a pass cannot do without -----------------------------------------------------------------------
def _payload_bytes(m, k, bits):
    return m * k * bits // 8 + m * (2 << bits)


def work(case):
    c = case
    if c["kind"] == "mlp":
        h, inter, bits = c["hidden"], c["inter"], c["bits"]
        return {"bytes": 2 * _payload_bytes(inter, h, bits) + _payload_bytes(h, inter, bits) + 4 * h, "flops": 6 * h * inter}
    if c["kind"] == "gemm":
        m, k, t = c["rows"], c["k"], c["tokens"]
        return {"bytes": _payload_bytes(m, k, c["bits"]) + 2 * t * (m + k), "flops": 2 * m * k * t}
    if c["kind"] == "quantise":  # read the matrix, write palettes and indices; one comparison per entry and value
        m, k = c["rows"], c["cols"]
        return {"bytes": 4 * m * k + _payload_bytes(m, k, 4), "flops": 16 * m * k}
    B, P, n = c["batch"], c["prompt"], c["new"] if c["kind"] == "generate" else c["steps"]
    if c["kind"] == "generate":
        h, qd, kvd, inter, L, bits = c["hidden"], c["heads"] * c["head_dim"], c["kv_heads"] * c["head_dim"], c["inter"], c["layers"], c["bits"]
        mats = [(qd + 2 * kvd, h), (h, qd), (2 * inter, h), (h, inter)]
        layer = sum(_payload_bytes(m, k, bits) for m, k in mats)
        head = _payload_bytes(c["vocab"], h, bits)
        seen = sum(range(P + 1, P + n + 1))  # cached positions read by the decode steps of a sequence
        params = sum(m * k for m, k in mats)
        pairs = P * (P + 1) // 2 + seen
        return {"bytes": L * layer * (n + (P > 0)) + n * head + L * 4 * kvd * B * (seen + P),
                "flops": 2 * L * params * B * (P + n) + 2 * c["vocab"] * h * B * n + 4 * L * qd * B * pairs}
    lens = [len(p) for p, _ in _trace_tokens(c, 0)]
    total, cfg = sum(lens), prism.LayeredConfig.from_dict(_layered_raw(c))
    size = 2 if c["dtype"] == "bfloat16" else 4
    dense = experts = 0
    for name, shape in cfg.tensor_shapes().items():
        if len(shape) != 2 or name in ("embed", "head", "pos"):
            continue
        if ".mlp.e" in name:
            experts += shape[0] * shape[1]
        else:
            dense += shape[0] * shape[1]
    used = lambda tokens: experts * min(1.0, tokens * 4 / 16)  # noqa: E731
    head = c["vocab"] * c["hidden"]
    bytes_ = 2 * (dense + used(total) + head) + n * 2 * (dense + used(B) + head) + 4 * c["vocab"] * B * (n + 1)
    qd = c["heads"] * c["head_dim"]
    pairs = sum(t * (t + 1) // 2 for t in lens) + sum(t + i for t in lens for i in range(1, n + 1))
    attn = 4 * qd * pairs * (c["layers"] if c["design"] == "tozarax" else c["layers"] // 2)
    linear_mix = 4 * qd * c["head_dim"] * (total + B * n) * (c["layers"] if c["design"] == "tozarax" else c["layers"] - c["layers"] // 2)
    state = size * c["layers"] * qd * B * n
    return {"bytes": int(bytes_ + state), "flops": int(2 * (dense + experts / 4) * (total + B * n) + 2 * head * B * (n + 1) + attn + linear_mix)}


def tolerance(case):
    if case["kind"] == "quantise":
        return "exact"
    if case["kind"] in ("mlp", "gemm"):
        return {"rel": 1e-3}
    if case["kind"] == "generate":
        return {"rel": 6e-3, "max": 0.1, "differ": 0.002}
    return {"rel": 3e-2 if case["dtype"] == "bfloat16" else 1e-4, "max": 0.5 if case["dtype"] == "bfloat16" else 1e-2}


# ---- the same in 64 bits -------------------------------------------------------------------------------
def exact(case, seed):
    c = case
    if c["kind"] == "quantise":
        return None  # bytes: nothing rounded in between
    if c["kind"] == "mlp":
        h, inter = c["hidden"], c["inter"]
        g, u, d = (_dense64(*_palette_and_index(m, k, c["bits"], k ** -0.5, seed, i)) for i, (m, k) in enumerate(((inter, h), (inter, h), (h, inter))))
        x = torch.randn(h, device="cuda", generator=_rand(seed, 9)).half().double()
        return d @ (torch.nn.functional.silu(g @ x) * (u @ x))
    if c["kind"] == "gemm":
        w = _dense64(*_palette_and_index(c["rows"], c["k"], c["bits"], c["k"] ** -0.5, seed))
        return torch.randn(c["tokens"], c["k"], device="cuda", generator=_rand(seed, 9)).half().double() @ w.T
    return _exact_generate(c, seed) if c["kind"] == "generate" else _exact_trace(c, seed)


def _rms(x, eps=EPS):
    return x / (x.square().mean(-1, keepdim=True) + eps).sqrt()


def _attend(q, k, v, scale, window=0):
    """Causal softmax attention of one sequence, q [T, H, D], k and v [T, G, .]: heads of a group share its keys."""
    T, H, G = q.shape[0], q.shape[1], k.shape[1]
    out = torch.empty(T, H, v.shape[2], dtype=torch.float64, device="cuda")
    at = torch.arange(T, device="cuda")
    for r in range(0, T, 2048):
        hi = min(T, r + 2048)
        lo = max(0, r - window + 1) if window else 0
        away = at[r:hi, None] - at[None, lo:hi]
        hide = (away < 0) | (away >= window) if window else away < 0
        for n in range(H):
            g = n // (H // G)
            p = (q[r:hi, n] @ k[lo:hi, g].T * scale).masked_fill_(hide, -math.inf).softmax(-1)
            out[r:hi, n] = p @ v[lo:hi, g]
    return out


def _exact_generate(c, seed):
    _, make = _model_tensors(c, seed)
    prompts, P, n, B = torch.from_numpy(_prompts(c, seed).astype(np.int64)).cuda(), c["prompt"], c["new"], c["batch"]
    nh, nkv, hd = c["heads"], c["kv_heads"], c["head_dim"]
    embed_pal, embed_idx = make("embed", 0)
    head = _dense64(*(make("embed", 0) if c["tied"] else make("lm_head", 0)))
    ang = torch.arange(P + n, device="cuda", dtype=torch.float64)[:, None] * THETA ** (-2.0 * torch.arange(hd // 2, device="cuda", dtype=torch.float64) / hd)
    cos, sin = ang.cos()[:, None], ang.sin()[:, None]

    def turn(x):
        a, b = x[..., :hd // 2], x[..., hd // 2:]
        return torch.cat([a * cos - b * sin, a * sin + b * cos], -1)

    # The prompt's last token is fed again as the first step's token; every step's token is the greedy choice before it.
    # All positions go through the model at once with assumed tokens, until the choices are the assumed ones.
    moved = torch.arange(n, device="cuda")[None] * (0 if c["tied"] else 1)
    fed = (prompts[:, -1:] + moved) % c["vocab"]
    for _ in range(4):
        x = _dense64(embed_pal, embed_idx)[torch.cat([prompts, fed], 1)]
        for layer in range(c["layers"]):
            w = lambda role: _dense64(*make(role, layer)).T  # noqa: E731
            a = _rms(x)
            q, k, v = a @ w("q"), a @ w("k"), a @ w("v")
            att = torch.stack([_attend(turn(q[b].view(-1, nh, hd)), turn(k[b].view(-1, nkv, hd)), v[b].view(-1, nkv, hd), hd ** -0.5) for b in range(B)])
            x = x + att.flatten(2) @ w("o")
            a = _rms(x)
            x = x + (torch.nn.functional.silu(a @ w("gate")) * (a @ w("up"))) @ w("down")
        logits = _rms(x[:, P:]) @ head.T
        tokens = logits.argmax(-1)
        if torch.equal(fed[:, 1:], tokens[:, :-1]):
            return {"tokens": tokens.cpu().numpy().astype(np.uint32), "logits": logits[:, -1].cpu().numpy()}
        fed = torch.cat([prompts[:, -1:], tokens[:, :-1]], 1)
    return None


def _exact_trace(c, seed):
    raw, tokens = _layered_raw(c), _trace_tokens(c, seed)
    w = {k: v.double() for k, v in _layered_weights(c, seed).items()}
    per_seq = []
    for prompt, after in tokens:
        t = torch.from_numpy(np.concatenate([prompt, after]).astype(np.int64)).cuda()
        x = (_mefipel64 if c["design"] == "mefipel" else _tozarax64)(raw, w, t)
        per_seq.append(x[len(prompt) - 1:] @ w["head"].T)
    return torch.stack(per_seq, 1).flatten(0, 1).cpu().numpy()


def _yarn64(rot):
    dims, base, sc = rot["dims"], rot["base"], rot["scaling"]
    pair = lambda turns: dims * math.log(sc["original"] / (2 * math.pi * turns)) / (2 * math.log(base))  # noqa: E731
    i = torch.arange(dims // 2, dtype=torch.float64, device="cuda")
    lo, hi = max(math.floor(pair(sc["fast"])), 0), min(math.ceil(pair(sc["slow"])), dims - 1)
    ramp = ((i - lo) / max(hi - lo, 0.001)).clamp(0, 1)
    freq = base ** (-2.0 * i / dims)
    return freq * (1 - ramp) + freq / sc["factor"] * ramp, 0.1 * math.log(sc["factor"]) + 1.0


def _mefipel64(raw, w, t):
    x, eps, T = w["embed"][t], raw["norm"]["eps"], len(t)
    at = torch.arange(T, device="cuda", dtype=torch.float64)
    for i, ly in enumerate(raw["layers"]):
        m, W = ly["mixer"], lambda n: w["l%d.%s" % (i, n)]  # noqa: B023, E731
        H, D, V = m["heads"], m["dim"], m["vdim"]
        h = _rms(x, eps) * W("norm1")
        gate = (h @ W("mix.g").T).sigmoid()
        if ly["type"] == "lightning":
            q, k = (torch.nn.functional.silu(h @ W("mix." + n).T).view(T, H, D) for n in "qk")
            v = torch.nn.functional.silu(h @ W("mix.v").T).view(T, H, V)
            away = at[:, None] - at[None]
            o = torch.empty(T, H, V, dtype=torch.float64, device="cuda")
            for n in range(H):
                decay = float(np.float32(m["decay"][n]))
                o[:, n] = ((q[:, n] @ k[:, n].T) * torch.where(away >= 0, decay ** away.clamp(min=0), 0.0)) @ v[:, n]
            o = _rms(o.flatten(1), eps) * W("mix.norm") * gate
        else:
            freq, mul = _yarn64(m["rot"])
            ang = at[:, None] * freq.float().double()
            cos, sin, half, R = (ang.cos() * mul)[:, None], (ang.sin() * mul)[:, None], m["rot"]["dims"] // 2, m["rot_dim"]

            def turn(z):
                a, b = z[..., :half], z[..., half:2 * half]
                return torch.cat([a * cos - b * sin, a * sin + b * cos, z[..., 2 * half:]], -1)  # noqa: B023

            q = ((_rms(h @ W("mix.dq").T, eps) * W("mix.dq.norm")) @ W("mix.uq").T).view(T, H, D + R)
            down = h @ W("mix.dkv").T
            lat = _rms(down[:, :m["kv_rank"]], eps) * W("mix.dkv.norm")
            k_rot = turn(down[:, None, m["kv_rank"]:]).expand(T, H, R)
            k = torch.cat([(lat @ W("mix.uk").T).view(T, H, D), k_rot], -1)
            q = torch.cat([q[..., :D], turn(q[..., D:])], -1)
            o = _attend(q, k, (lat @ W("mix.uv").T).view(T, H, V), m["scale"], m["mask"]["size"]).flatten(1) * gate
        up = torch.nn.functional.gelu(h @ W("mlp.up").T + W("mlp.up.b"), approximate="tanh")
        x = x + raw["residual_mult"] * (o @ W("mix.o").T + up @ W("mlp.down").T + W("mlp.down.b"))
    return _rms(x, eps) * w["final.norm"] * raw["logit_scale"]


def _conv64(x, taps):
    n = taps.shape[1]
    padded = torch.cat([x.new_zeros(n - 1, x.shape[1]), x])
    return sum(padded[j:j + x.shape[0]] * taps[:, j] for j in range(n))


def _tozarax64(raw, w, t):
    eps, T = raw["norm"]["eps"], len(t)
    silu, x = torch.nn.functional.silu, w["embed"][t] + w["pos"][:T]
    history = [x]
    for i, ly in enumerate(raw["layers"]):
        W, left, right = lambda n: w["l%d.%s" % (i, n)], ly["mixer"]["left"], ly["mixer"]["right"]  # noqa: B023, E731

        def sub(x, n, f):
            h = _rms(x, eps) * (1.0 + W("norm" + n))
            return x + f(h + _conv64(h, W("canon" + n))) * (h @ W("rg" + n).T + W("rg" + n + ".b")).sigmoid()

        def mixer(h):
            H, G, D = left["heads"], left["kv_heads"], left["dim"]
            q, k, v = ((h @ W("mix.left." + n).T).view(T, g, D) for n, g in (("q", H), ("k", G), ("v", G)))
            a = _attend(q, k, v, left["scale"], left["mask"]["size"]).flatten(1) @ W("mix.left.o").T
            H, G, D, V = right["heads"], right["kv_heads"], right["dim"], right["vdim"]
            q, k, v = (silu(_conv64(h @ W("mix.right." + n).T, W("mix.right." + n + ".conv"))) for n in "qkv")
            unit = lambda z: z / (z.square().sum(-1, keepdim=True) + 1e-6).sqrt()  # noqa: E731
            q, k = (unit(z.view(T, G, D)).repeat_interleave(H // G, 1) for z in (q, k))
            v, q = v.view(T, H, V), q * D ** -0.5
            beta = (h @ W("mix.right.b").T).sigmoid()
            decay = (-W("mix.right.A_log").exp() * torch.nn.functional.softplus(h @ W("mix.right.a").T + W("mix.right.dt_bias"))).exp()
            S, o = x.new_zeros(H, D, V), x.new_empty(T, H, V)
            for j in range(T):
                S = S * decay[j, :, None, None]
                u = beta[j, :, None] * (v[j] - torch.einsum("hd,hdv->hv", k[j], S))
                S = S + k[j, :, :, None] * u[:, None, :]
                o[j] = torch.einsum("hd,hdv->hv", q[j], S)
            o = _rms(o, eps) * W("mix.right.norm") * silu(h @ W("mix.right.g").T).view(T, H, V)
            b = o.flatten(1) @ W("mix.right.o").T
            return 0.5 * (_rms(a, eps) * W("mix.left.out") + _rms(b, eps) * W("mix.right.out"))

        def experts(h):
            r = ly["mlp"]["router"]
            score = (h @ W("mlp.router").T).sigmoid()
            choice, groups = score + W("mlp.correction"), r["groups"]
            best = choice.view(T, groups["count"], -1).topk(2, -1).values.sum(-1).topk(groups["keep"], -1).indices
            keep = torch.zeros(T, groups["count"], device="cuda").scatter_(1, best, 1.0).repeat_interleave(r["experts"] // groups["count"], 1)
            chosen = choice.masked_fill(keep == 0, -math.inf).topk(r["top"], -1).indices
            y = torch.zeros_like(h)
            for e in range(r["experts"]):
                rows = (chosen == e).any(1).nonzero().flatten()
                if len(rows):
                    up = (h[rows] @ W("mlp.e%d.up" % e).T).clamp(min=0).square()
                    y[rows] += score[rows, e, None] * (up @ W("mlp.e%d.down" % e).T)
            return y

        x = sub(sub(x, "1", mixer), "2", experts)
        history.append(x)
        x = sum(a * z for a, z in zip(W("dwa"), history))
    return _rms(x, eps) * (1.0 + w["final.norm"])
