"""What a step of the engine is made of, as cases whose time can be measured and whose results can be compared.

Most cases are one layer part each (a mixer or a feed-forward, called through `Part.forward` over a step that the cache
manager laid out), at the layer sizes of `bench.py`; two are whole: a 32-bit feed-forward as replay in 32-bit runs it, and
a model that is fed two prompts and then decodes.  A step of single tokens is captured in a CUDA graph once and replayed,
as the engine does with its decode steps; a step with portions of prompts is launched from Python.
"""
from __future__ import annotations

import math

import torch

from fastmlx_b200.cache import CacheManager
from fastmlx_b200.engine.batch import StepEntry, build_context
from fastmlx_b200.engine.loading import make_runtime, random_model
from fastmlx_b200.engine.step import StepFunction
from fastmlx_b200.parts import (ChannelDeltaMixer, GatedDeltaMixer, GQAAttention, PairMixer, RetentionMixer, RotaryEmbedding,
                                RoutedExperts, StateSpaceMixer, SwiGLU)

F64 = torch.float64
SIZES = {"1b": dict(width=2048, heads=32, kv_heads=8, dim=64, ff=8192),
         "8b": dict(width=4096, heads=32, kv_heads=8, dim=128, ff=14336)}
PAGE, THETA, EPS, TAPS = 16, 500000.0, 1e-6, 4
WINDOW, CAP = 1024, 30.0
SSM_STATE, SSM_VDIM, SSM_GROUPS = 128, 64, 8
EXPERTS, TOP = 16, 4
VOCAB, LAYERS = 128256, 4
RECURRENT = ("delta", "channel", "ssm", "pair")


# ----------------------------------------------------------------------------- the cases
def listed():
    return [
        # one request decodes: the feed-forward of a small model, bound by launch and the stream of weights
        dict(name="mlp-decode-1b", kind="mlp", size="1b", rows=1, tokens=1, context=0, dtype="bfloat16"),
        # replay in 32-bit, which must give the same bits however a prompt is cut: its products, an odd portion
        dict(name="mlp-portion-32bit-1b", kind="mlp", size="1b", rows=1, tokens=333, context=0, dtype="float32"),
        # the flagship's headline: eight requests decode behind long contexts
        dict(name="attention-decode-1b", kind="attention", size="1b", rows=8, tokens=8, context=8192, dtype="bfloat16"),
        # a whole prompt of the larger dense model
        dict(name="attention-prompt-8b", kind="attention", size="8b", rows=1, tokens=2048, context=0, dtype="bfloat16"),
        # later portions of three prompts in one step: sliding window, q/k norm, capped scores
        dict(name="window-portions-1b", kind="window", size="1b", rows=3, tokens=2499, context=700, dtype="bfloat16"),
        # a prompt through a layer with a gated delta rule, and 64 requests that decode through it
        dict(name="delta-prompt-1b", kind="delta", size="1b", rows=1, tokens=2048, context=0, dtype="bfloat16"),
        dict(name="delta-decode-1b", kind="delta", size="1b", rows=64, tokens=64, context=300, dtype="bfloat16"),
        # five ragged prompts through a state-space layer
        dict(name="ssm-prompts-1b", kind="ssm", size="1b", rows=5, tokens=1777, context=0, dtype="bfloat16"),
        # a prompt through the pair of sigmoid attention with mixed heads and a retention
        dict(name="pair-prompt-1b", kind="pair", size="1b", rows=1, tokens=1531, context=0, dtype="bfloat16"),
        # two prompts through a delta rule with a decay per key channel, at the larger model's sizes
        dict(name="channel-prompts-8b", kind="channel", size="8b", rows=2, tokens=2048, context=0, dtype="bfloat16"),
        # a portion through a mixture of experts
        dict(name="experts-portion-1b", kind="experts", size="1b", rows=1, tokens=1024, context=0, dtype="bfloat16"),
        # a whole call: two prompts in one step, then both decode
        dict(name="model-1b", kind="model", size="1b", rows=2, tokens=700, context=0, dtype="bfloat16", decode=12),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """A case of the same parts: a step of one token for each of up to 64 requests, or one with up to 2,048 tokens of up to
    six prompts; behind no context or up to 8,192 tokens of it."""
    kind = rng.choice(["mlp", "attention", "window", "delta", "ssm", "pair", "channel", "experts", "model"])
    size = "1b" if kind in ("pair", "model") else rng.choice(["1b", "1b", "8b"])
    dtype = "float32" if kind == "mlp" and rng.random() < 0.4 else "bfloat16"
    if kind == "model":
        rows = rng.randint(1, 6)
        return dict(kind=kind, size=size, rows=rows, tokens=rows * _log(rng, 8, 150), context=0, dtype=dtype, decode=rng.randint(2, 12))
    most = {"pair": 1531, "mlp": 2048 if dtype == "bfloat16" else 333}.get(kind, 2048)
    if rng.random() < 0.35:
        rows = _log(rng, 1, 64)
        context = _log(rng, 16, 8192 if rows <= 8 else 1024)
        return dict(kind=kind, size=size, rows=rows, tokens=rows, context=context, dtype=dtype)
    tokens = _log(rng, 20, most)
    rows = rng.randint(1, min(6, tokens // 8))
    context = _log(rng, 16, 1500) if kind != "pair" and rng.random() < 0.4 else 0
    return dict(kind=kind, size=size, rows=rows, tokens=tokens, context=context, dtype=dtype)


def _portions(case):
    """Tokens that each row brings: one each, or shares of the step's tokens that differ from row to row."""
    R, T = case["rows"], case["tokens"]
    if T == R:
        return [1] * R
    share = [3 + 2 * (i % 3) for i in range(R)]
    out = [max(1, T * s // sum(share)) for s in share]
    out[-1] += T - sum(out)
    return out


def _contexts(case):
    """Tokens of each row that are in the cache already: up to the case's number, not all the same."""
    return [case["context"] - (case["context"] // 9) * (i % 4) for i in range(case["rows"])]


def _decode(case):
    return case["tokens"] == case["rows"]


# ----------------------------------------------------------------------------- inputs
def _names(case):
    """The tensors of the case's part: (name, shape, kind of values)."""
    s, kind = SIZES[case["size"]], case["kind"]
    d, H, G, D = s["width"], s["heads"], s["kv_heads"], s["dim"]
    if kind == "mlp":
        return [("m.gate.weight", (s["ff"], d), "matrix"), ("m.up.weight", (s["ff"], d), "matrix"), ("m.down.weight", (d, s["ff"]), "matrix")]
    if kind in ("attention", "window"):
        out = [("m.q.weight", (H * D, d), "matrix"), ("m.k.weight", (G * D, d), "matrix"), ("m.v.weight", (G * D, d), "matrix"),
               ("m.o.weight", (d, H * D), "matrix")]
        return out if kind == "attention" else out + [(n.replace("weight", "bias"), sh[:1], "bias") for n, sh, _ in out]
    if kind == "delta":
        return [("m.q.weight", (G * D, d), "matrix"), ("m.k.weight", (G * D, d), "matrix"), ("m.v.weight", (H * D, d), "matrix"),
                ("m.g.weight", (H * D, d), "matrix"), ("m.b.weight", (H, d), "matrix"), ("m.a.weight", (H, d), "matrix"),
                ("m.o.weight", (d, H * D), "matrix"), ("m.q.conv", (G * D, TAPS), "conv"), ("m.k.conv", (G * D, TAPS), "conv"),
                ("m.v.conv", (H * D, TAPS), "conv"), ("m.A_log", (H,), "log_rate"), ("m.dt_bias", (H,), "rate_bias"), ("m.norm", (D,), "norm")]
    if kind == "channel":
        r = d // 128 * 8
        return [("m.q.weight", (G * D, d), "matrix"), ("m.k.weight", (G * D, d), "matrix"), ("m.v.weight", (H * D, d), "matrix"),
                ("m.a1.weight", (r, d), "matrix"), ("m.g1.weight", (r, d), "matrix"), ("m.b.weight", (H, d), "matrix"),
                ("m.a2.weight", (H * D, r), "matrix"), ("m.g2.weight", (H * D, r), "matrix"), ("m.o.weight", (d, H * D), "matrix"),
                ("m.q.conv", (G * D, TAPS), "conv"), ("m.k.conv", (G * D, TAPS), "conv"), ("m.v.conv", (H * D, TAPS), "conv"),
                ("m.A_log", (H,), "log_rate"), ("m.dt_bias", (H * D,), "rate_bias"), ("m.norm", (D,), "norm")]
    if kind == "ssm":
        Hs = 2 * d // SSM_VDIM
        inner, gn = Hs * SSM_VDIM, SSM_GROUPS * SSM_STATE
        return [("m.in", (2 * inner + 2 * gn + Hs, d), "matrix"), ("m.conv", (inner + 2 * gn, TAPS), "conv"), ("m.conv.b", (inner + 2 * gn,), "bias"),
                ("m.dt_bias", (Hs,), "rate_bias"), ("m.A_log", (Hs,), "log_rate"), ("m.D", (Hs,), "norm"), ("m.norm", (inner,), "norm"),
                ("m.o", (d, inner), "matrix")]
    if kind == "pair":
        return [("m.left.q", (H * D, d), "matrix"), ("m.left.k", (G * D, d), "matrix"), ("m.left.v", (G * D, d), "matrix"),
                ("m.left.o", (d, H * D), "matrix"), ("m.left.q.norm", (H * D,), "norm"), ("m.left.k.norm", (G * D,), "norm"),
                ("m.left.talk", (H, H), "head_mix"), ("m.left.pb", (H,), "head_bias"), ("m.right.q", (H * D, d), "matrix"),
                ("m.right.k", (H * D, d), "matrix"), ("m.right.v", (H * D, d), "matrix"), ("m.right.g", (H * D, d), "matrix"),
                ("m.right.o", (d, H * D), "matrix"), ("m.left.out", (d,), "norm"), ("m.right.out", (d,), "norm")]
    ff = s["ff"] // 4                                                       # experts
    out = [("m.router", (EXPERTS, d), "matrix"), ("m.router.b", (EXPERTS,), "bias")]
    for e in range(EXPERTS):
        out += [(f"m.e{e}.gate", (ff, d), "matrix"), (f"m.e{e}.up", (ff, d), "matrix"), (f"m.e{e}.down", (d, ff), "matrix")]
    return out


def _values(shape, kind, g):
    """Weights as random models of this package have them: matrices N(0, 0.02), norms around one, convolution taps of the order of
    one, decays spread over (0, 1), mixes of heads near the identity, sigmoid weights well below one."""
    t = torch.randn(shape, generator=g, device="cuda")
    if kind == "conv":
        t = t * 0.5
    elif kind == "log_rate":
        t = torch.log(torch.sigmoid(t) * 0.98 + 0.02)
    elif kind == "rate_bias":
        t = t * 0.5 - 1.0
    elif kind == "head_mix":
        t = torch.eye(shape[0], device="cuda") + t * 0.1
    elif kind == "head_bias":
        t = t * 0.5 - 3.0
    else:
        t = t * 0.02 + (1.0 if kind == "norm" else 0.0)
    return t.bfloat16()


def _state_floats(case):
    """Floats of a recurrent part's slot per request: the matrices of state, and all of it (the convolution's last inputs too)."""
    s, kind = SIZES[case["size"]], case["kind"]
    H, G, D = s["heads"], s["kv_heads"], s["dim"]
    if kind == "ssm":
        Hs = 2 * s["width"] // SSM_VDIM
        S, C = Hs * SSM_VDIM * SSM_STATE, Hs * SSM_VDIM + 2 * SSM_GROUPS * SSM_STATE
    elif kind == "pair":
        S, C = H * D * D, 0
    else:
        S, C = H * D * D, 2 * G * D + H * D
    return S, S + (TAPS - 1) * C


def _inputs(case, seed):
    """Everything random, from the seed alone: weights by name, the step's normalised activations, and what earlier steps left
    (keys and values per row, or the slots of state)."""
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    s = SIZES[case["size"]]
    W = {n: _values(sh, kind, g) for n, sh, kind in _names(case)}
    dt = torch.float32 if case["dtype"] == "float32" else torch.bfloat16
    x = torch.randn(case["tokens"], s["width"], generator=g, device="cuda").to(dt)
    past = [torch.randn(c, 2, s["kv_heads"], s["dim"], generator=g, device="cuda").bfloat16() for c in _contexts(case)] \
        if case["kind"] in ("attention", "window", "pair") else None
    state = None
    if case["kind"] in RECURRENT:
        state = torch.randn(case["rows"], _state_floats(case)[1], generator=g, device="cuda") * (0.1 if case["context"] else 0.0)
    return W, x, past, state


def _decays(heads):
    return [1.0 - 2.0 ** -(5 + 3 * i / (heads - 1)) for i in range(heads)]


def _part(case):
    s, kind = SIZES[case["size"]], case["kind"]
    d, H, G, D = s["width"], s["heads"], s["kv_heads"], s["dim"]
    if kind == "mlp":
        return SwiGLU(d, s["ff"], "m", proj_names=("gate", "up", "down"))
    if kind == "attention":
        return GQAAttention(d, H, G, D, RotaryEmbedding(D, THETA), "m", proj_names=("q", "k", "v", "o"))
    if kind == "window":
        return GQAAttention(d, H, G, D, RotaryEmbedding(D, THETA, rotary_dim=D // 2), "m", bias=True, window=WINDOW, softcap=CAP,
                            qk_norm_eps=EPS, proj_names=("q", "k", "v", "o"))
    if kind == "delta":
        return GatedDeltaMixer(d, H, G, D, D, TAPS, EPS, "m")
    if kind == "channel":
        return ChannelDeltaMixer(d, H, G, D, D, TAPS, EPS, "m")
    if kind == "ssm":
        return StateSpaceMixer(d, 2 * d // SSM_VDIM, SSM_VDIM, SSM_STATE, SSM_GROUPS, SSM_GROUPS, TAPS, EPS, "m")
    if kind == "pair":
        left = GQAAttention(d, H, G, D, RotaryEmbedding(D, THETA), "m.left", softcap=CAP, qk_norm_eps=EPS, qk_norm_weights=("q.norm", "k.norm"),
                            qk_norm_first=True, qk_norm_whole=True, weights="sigmoid", head_bias="pb", head_mix="talk",
                            proj_names=("q", "k", "v", "o"), weight_suffix="")
        right = RetentionMixer(d, H, D, D, _decays(H), EPS, "m.right", rot_dims=D, rot_base=THETA)
        return PairMixer(d, left, right, EPS, "m")
    return RoutedExperts(d, EXPERTS, TOP, s["ff"] // 4, 0.0, "m", activation="silu", router_bias="router.b", weights="chosen")


# ----------------------------------------------------------------------------- one pass
def _tokens(case, seed):
    """Prompts and the tokens that are fed one by one after them."""
    g = torch.Generator()
    g.manual_seed(int(seed) + 1)
    return [torch.randint(0, VOCAB, (n + case["decode"],), generator=g).tolist() for n in _portions(case)]


def _prepare_model(case, seed):
    s = SIZES[case["size"]]
    cfg = dict(model_type="llama", architectures=["LlamaForCausalLM"], num_hidden_layers=LAYERS, hidden_size=s["width"],
               num_attention_heads=s["heads"], num_key_value_heads=s["kv_heads"], head_dim=s["dim"], intermediate_size=s["ff"],
               vocab_size=VOCAB, rope_theta=THETA, rms_norm_eps=1e-5, tie_word_embeddings=True, max_position_embeddings=131072)
    _, model, rt = random_model(cfg, int(seed))
    tokens = _tokens(case, seed)
    manager = CacheManager(model.cache_needs(), page_size=PAGE, num_pages=sum(-(-len(t) // PAGE) for t in tokens) + 1,
                           max_requests=case["rows"], dtype=rt.dtype, device=rt.device)
    return dict(case=case, fn=StepFunction(model, manager, rt, cuda_graphs=True), manager=manager, tokens=tokens)


def prepare(case, seed):
    if case["kind"] == "model":
        return _prepare_model(case, seed)
    W, x, past, state = _inputs(case, seed)
    rt = make_runtime(case["dtype"])
    part = _part(case)
    part.bind(W, rt)
    if case["kind"] in ("mlp", "experts"):
        st = dict(case=case, part=part, args=(x, None), state=None, keep=None)
    else:
        q, c = _portions(case), _contexts(case)
        pages = sum(-(-(a + b) // PAGE) + 1 for a, b in zip(q, c))
        manager = CacheManager([(part.cache_spec(), part.state_spec(), None)], page_size=PAGE, num_pages=pages, max_requests=case["rows"],
                               dtype=rt.dtype, device=rt.device)
        cache, entries = manager.entries[0], []
        for r in range(case["rows"]):
            req = manager.add_request(r)
            if c[r]:
                manager.reserve(req, c[r])
                if past is not None:
                    ids = torch.tensor(req.tables[0].pages, device="cuda")
                    kv = torch.cat([past[r], past[r].new_zeros(len(ids) * PAGE - c[r], *past[r].shape[1:])])
                    held = ids >= 0                     # pages that a window has not given back
                    cache.kv[ids[held]] = kv.view(len(ids), PAGE, *kv.shape[1:]).permute(0, 2, 3, 1, 4)[held]
                manager.commit(req)
            if state is not None:
                cache.state[req.slot, :state.shape[1]] = state[r]
            manager.reserve(req, q[r])
            entries.append(StepEntry(req, [0] * q[r], []))
        ctx = build_context(entries, manager, rt.device, torch.zeros(4, dtype=torch.int32, device=rt.device))
        slots = cache.state[[e.request.slot for e in entries]] if state is not None else None
        st = dict(case=case, part=part, args=(x, ctx, cache), state=None, keep=(manager, slots))
        if state is not None:
            assert [e.request.slot for e in entries] == list(range(case["rows"]))
            st["state"] = cache.state
    if _decode(case):                                   # captured once; what the warm-up did to the slots is undone
        part.forward(*st["args"])
        torch.cuda.synchronize()
        st["graph"] = torch.cuda.CUDAGraph()
        with torch.cuda.graph(st["graph"]):
            st["out"] = part.forward(*st["args"])
        if st["state"] is not None:
            st["state"][:case["rows"]] = st["keep"][1]
    return st


def run(state):
    case = state["case"]
    if case["kind"] == "model":
        fn, manager, n = state["fn"], state["manager"], case["decode"]
        reqs = [manager.add_request(r) for r in range(case["rows"])]
        logits = [fn.run([StepEntry(q, t[:len(t) - n], [len(t) - n - 1]) for q, t in zip(reqs, state["tokens"])], check=False)]
        for i in range(n, 0, -1):
            logits.append(fn.run([StepEntry(q, [t[-i]], [0]) for q, t in zip(reqs, state["tokens"])], check=False).clone())
        for r in range(case["rows"]):
            manager.free(r)
        return logits
    if "graph" in state:
        state["graph"].replay()
        out = state["out"]
    else:
        out = state["part"].forward(*state["args"])
    return out if state["state"] is None else (out, state["state"])


# ----------------------------------------------------------------------------- what a pass cannot do without
def _pairs(case, window=0):
    """(query, key) pairs in sight."""
    n = 0
    for q, c in zip(_portions(case), _contexts(case)):
        if not window:
            n += q * c + q * (q + 1) // 2
        else:
            n += sum(min(p + 1, window) for p in range(c, c + q))
    return n


def work(case):
    s, kind, T = SIZES[case["size"]], case["kind"], case["tokens"]
    d, H, G, D = s["width"], s["heads"], s["kv_heads"], s["dim"]
    e = 4 if case["dtype"] == "float32" else 2
    if kind == "model":
        layer = d * (H + 2 * G) * D + H * D * d + 3 * d * s["ff"]
        toks = T + case["rows"] * case["decode"]
        return {"bytes": float(2 * (LAYERS * layer + VOCAB * d) * (case["decode"] + 1)),
                "flops": 2.0 * toks * LAYERS * layer + 2.0 * case["rows"] * (case["decode"] + 1) * VOCAB * d + 4.0 * LAYERS * H * D * _pairs(case)}
    weights = sum(math.prod(sh) for _, sh, k in _names(case) if k == "matrix")
    flops = 2.0 * T * weights
    if kind == "experts":
        one = 3 * d * (s["ff"] // 4)
        weights = EXPERTS * d + min(EXPERTS, TOP * T) * one
        flops = 2.0 * T * (EXPERTS * d + TOP * one)
    nbytes = weights * e + 2 * T * d * e
    if kind in ("attention", "window", "pair"):
        n = _pairs(case, WINDOW if kind == "window" else 0)
        flops += 4.0 * H * D * n + (2.0 * H * H * n if kind == "pair" else 0.0)
        seen = sum(min(c, WINDOW) if kind == "window" else c for c in _contexts(case))
        nbytes += (seen + T) * 2 * G * D * 2
    if kind in RECURRENT:
        S = _state_floats(case)[0]
        flops += T * S * (4.0 if kind in ("ssm", "pair") else 6.0)
        nbytes += 2 * case["rows"] * _state_floats(case)[1] * 4
    return {"bytes": float(nbytes), "flops": flops}


def tolerance(case):
    """bfloat16 activations between a part's kernels: about four times what the parts show against 64-bit arithmetic (0.0023 to
    0.0041; attention over a whole prompt, whose queries and weights are bfloat16 too, 0.0055, and a model of four such layers).
    32-bit products: their order of summation (2e-6 over 8,192 terms)."""
    if case["dtype"] == "float32":
        return {"rel": 8e-6}
    return {"rel": 0.02 if case["kind"] in ("attention", "model") else 0.015}


# ----------------------------------------------------------------------------- the same in 64-bit
def _silu(z):
    return z * torch.sigmoid(z)


def _rms(z, eps=EPS):
    return z / torch.sqrt(z.square().mean(-1, keepdim=True) + eps)


def _turn(h, positions, dims):
    """h [T, heads, D] rotated over its first `dims` dimensions, i paired with i + dims / 2."""
    f = THETA ** (-torch.arange(0, dims, 2, dtype=F64, device=h.device) / dims)
    a = positions.to(F64)[:, None] * f
    c, s, m = a.cos()[:, None], a.sin()[:, None], dims // 2
    x, y = h[..., :m], h[..., m:dims]
    return torch.cat([x * c - y * s, y * c + x * s, h[..., dims:]], -1)


def _rows(case):
    at = 0
    for r, (q, c) in enumerate(zip(_portions(case), _contexts(case))):
        yield r, slice(at, at + q), torch.arange(c, c + q, device="cuda")
        at += q


def _conv(z, before, w, bias=None):
    """z [q, C] behind `before` [taps - 1, C] through a causal convolution per channel and SiLU -> (values, the last inputs)."""
    full = torch.cat([before, z])
    y = sum(full[j:j + len(z)] * w[:, j] for j in range(TAPS))
    return _silu(y if bias is None else y + bias), full[len(full) - (TAPS - 1):]


def _unit(z):
    return z / torch.sqrt(z.square().sum(-1, keepdim=True) + 1e-6)


def _softplus(z):
    return torch.nn.functional.softplus(z, threshold=60.0)


def _attend(q, k, v, qpos, case, W, pre=""):
    """q [q, H, D] over k, v [n, G, D], keys at positions 0 .. n-1."""
    kind, H, G = case["kind"], q.shape[1], k.shape[1]
    kpos = torch.arange(len(k), device=q.device)
    hidden = kpos[None] > qpos[:, None]
    if kind == "window":
        hidden |= kpos[None] <= qpos[:, None] - WINDOW
    out = []
    for g in range(G):
        s = torch.einsum("qhd,kd->hqk", q[:, g * (H // G):(g + 1) * (H // G)], k[:, g]) * q.shape[-1] ** -0.5
        if kind in ("window", "pair"):
            s = CAP * torch.tanh(s / CAP)
        if kind == "pair":
            s = torch.sigmoid(s + W["m.left.pb"][g * (H // G):(g + 1) * (H // G), None, None]).masked_fill(hidden, 0.0)
            out.append(s)
        else:
            out.append(torch.einsum("hqk,kd->qhd", torch.softmax(s.masked_fill(hidden, -math.inf), -1), v[:, g]))
    if kind != "pair":
        return torch.cat(out, 1)
    w = torch.cat(out)                                                       # [H, q, n]
    return torch.stack([torch.einsum("qk,kd->qd", torch.einsum("g,gqk->qk", W["m.left.talk"][h], w), v[:, h // (H // G)])
                        for h in range(H)], 1)


def _recur(q, k, v, decay, beta, S):
    """Tokens in order: S [H, D, P] decays (per head or per row of state), takes k v^T (with `beta`: the delta rule's write) and is
    read with q.  -> (o [T, H, P], S)."""
    out = torch.empty_like(v)
    for t in range(len(q)):
        S = S * (decay[t][:, None, None] if decay.dim() == 2 else decay[t][:, :, None])
        u = v[t] if beta is None else beta[t][:, None] * (v[t] - torch.einsum("hdp,hd->hp", S, k[t]))
        S = S + k[t][:, :, None] * u[:, None, :]
        out[t] = torch.einsum("hdp,hd->hp", S, q[t])
    return out, S


def _exact_attention(case, W, x, past, pre="m."):
    s = SIZES[case["size"]]
    H, G, D = s["heads"], s["kv_heads"], s["dim"]
    suffix = "" if case["kind"] == "pair" else ".weight"
    q, k, v = (x @ W[f"{pre}{n}{suffix}"].T for n in "qkv")
    if case["kind"] == "window":
        q, k, v = (t + W[f"{pre}{n}.bias"] for t, n in ((q, "q"), (k, "k"), (v, "v")))
    if case["kind"] == "pair":
        q, k = _rms(q) * W[pre + "q.norm"], _rms(k) * W[pre + "k.norm"]
    out = []
    for r, at, pos in _rows(case):
        dims = D // 2 if case["kind"] == "window" else D
        qr, kr = (_turn(t[at].view(-1, n, D), pos, dims) for t, n in ((q, H), (k, G)))
        if case["kind"] == "window":
            qr, kr = _rms(qr), _rms(kr)
        kk = torch.cat([past[r][:, 0].to(F64), kr])
        vv = torch.cat([past[r][:, 1].to(F64), v[at].view(-1, G, D)])
        out.append(_attend(qr, kk, vv, pos, case, W).reshape(-1, H * D))
    y = torch.cat(out) @ W[f"{pre}o{suffix}"].T
    return y + W[pre + "o.bias"] if case["kind"] == "window" else y


def _exact_delta(case, W, x, state):
    s = SIZES[case["size"]]
    H, G, D, n = s["heads"], s["kv_heads"], s["dim"], _state_floats(case)
    z = torch.cat([x @ W[f"m.{p}.weight"].T for p in "qkv"], 1)
    taps = torch.cat([W[f"m.{p}.conv"] for p in "qkv"])
    beta = torch.sigmoid(x @ W["m.b.weight"].T)
    if case["kind"] == "delta":
        decay = torch.exp(-torch.exp(W["m.A_log"]) * _softplus(x @ W["m.a.weight"].T + W["m.dt_bias"]))
        gate = _silu(x @ W["m.g.weight"].T)
    else:
        a = (x @ W["m.a1.weight"].T) @ W["m.a2.weight"].T + W["m.dt_bias"]
        decay = torch.exp(-torch.exp(W["m.A_log"])[:, None] * _softplus(a).view(-1, H, D))
        gate = torch.sigmoid((x @ W["m.g1.weight"].T) @ W["m.g2.weight"].T)
    out, left = [], state.to(F64).clone()
    for r, at, _ in _rows(case):
        y, last = _conv(z[at], state[r, n[0]:].to(F64).view(TAPS - 1, -1), taps)
        q, k, v = (t.view(len(y), -1, D) for t in y.split([G * D, G * D, H * D], 1))
        q, k = (_unit(t).repeat_interleave(H // G, 1) for t in (q, k))
        o, S = _recur(q * D ** -0.5, k, v, decay[at], beta[at], state[r, :n[0]].to(F64).view(H, D, D).transpose(1, 2))
        out.append((_rms(o) * W["m.norm"]).reshape(len(y), -1))
        left[r] = torch.cat([S.transpose(1, 2).reshape(-1), last.reshape(-1)])
    return (torch.cat(out) * gate) @ W["m.o.weight"].T, left


def _exact_ssm(case, W, x, state):
    H, G, N, P, n = 2 * SIZES[case["size"]]["width"] // SSM_VDIM, SSM_GROUPS, SSM_STATE, SSM_VDIM, _state_floats(case)
    z, xbc, dt = (x @ W["m.in"].T).split([H * P, H * P + 2 * G * N, H], 1)
    dt = _softplus(dt + W["m.dt_bias"])
    decay = torch.exp(-torch.exp(W["m.A_log"]) * dt)
    out, left = [], state.to(F64).clone()
    for r, at, _ in _rows(case):
        y, last = _conv(xbc[at], state[r, n[0]:].to(F64).view(TAPS - 1, -1), W["m.conv"], W["m.conv.b"])
        v, b, c = (t.view(len(y), -1, w) for t, w in zip(y.split([H * P, G * N, G * N], 1), (P, N, N)))
        b, c = (t.repeat_interleave(H // G, 1) for t in (b, c))
        o, S = _recur(c, b * dt[at][:, :, None], v, decay[at], None, state[r, :n[0]].to(F64).view(H, P, N).transpose(1, 2))
        out.append((o + W["m.D"][:, None] * v).reshape(len(y), -1))
        left[r] = torch.cat([S.transpose(1, 2).reshape(-1), last.reshape(-1)])
    y = torch.cat(out) * _silu(z)
    return (_rms(y.view(len(y), G, -1)).reshape(len(y), -1) * W["m.norm"]) @ W["m.o"].T, left


def _exact_pair(case, W, x, past, state):
    s = SIZES[case["size"]]
    H, D = s["heads"], s["dim"]
    a = _exact_attention(case, W, x, past, "m.left.")
    q, k, v, g = (x @ W[f"m.right.{p}"].T for p in "qkvg")
    decay = torch.tensor(_decays(H), dtype=F64, device="cuda")
    out, left = [], state.to(F64).clone()
    for r, at, pos in _rows(case):
        qr, kr = (_turn(t[at].view(-1, H, D), pos, D) for t in (q, k))
        o, S = _recur(qr, kr * D ** -0.5, v[at].view(-1, H, D), decay.expand(len(pos), H), None,
                      state[r].to(F64).view(H, D, D).transpose(1, 2))
        out.append(_rms(o).reshape(len(pos), -1))
        left[r] = S.transpose(1, 2).reshape(-1)
    b = (torch.cat(out) * _silu(g)) @ W["m.right.o"].T
    return (_rms(a) * W["m.left.out"] + _rms(b) * W["m.right.out"]) / 2, left


def exact(case, seed):
    if case["kind"] == "model":
        return None          # its weights are the engine's own random ones; its parts are compared one by one
    W, x, past, state = _inputs(case, seed)
    x, W = x.to(F64), ({n: t.to(F64) for n, t in W.items()} if case["kind"] != "experts" else W)
    if case["kind"] == "mlp":
        return (_silu(x @ W["m.gate.weight"].T) * (x @ W["m.up.weight"].T)) @ W["m.down.weight"].T
    if case["kind"] in ("attention", "window"):
        return _exact_attention(case, W, x, past)
    if case["kind"] in ("delta", "channel"):
        return _exact_delta(case, W, x, state)
    if case["kind"] == "ssm":
        return _exact_ssm(case, W, x, state)
    if case["kind"] == "pair":
        return _exact_pair(case, W, x, past, state)
    logits = x @ W["m.router"].to(F64).T + W["m.router.b"].to(F64)
    best, chosen = logits.topk(TOP, -1)
    share, y = torch.softmax(best, -1), torch.zeros_like(x)
    for e in range(EXPERTS):
        t, i = (chosen == e).nonzero(as_tuple=True)
        gate, up, down = (W[f"m.e{e}.{p}"].to(F64) for p in ("gate", "up", "down"))
        y[t] += share[t, i][:, None] * ((_silu(x[t] @ gate.T) * (x[t] @ up.T)) @ down.T)
    return y
