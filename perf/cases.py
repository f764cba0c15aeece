"""The work that programs have this package do, as cases that can be timed and compared with plain arithmetic.

Every case goes through the package's own entry points: ``Engine.step`` for whole calls, and the parts a model is put
together from (``ccinfer_b200.parts``), bound to a ``Runtime`` and called with a ``StepContext`` as the engine calls
them.  Layer sizes are those of ``bench.py``: width 2048 with 16 query and 8 key heads, and width 4096 with 32 and 8.

A part that gets a few single tokens is replayed from a CUDA graph, as the engine replays its decode steps; portions of
prompts are launched one kernel after the other, as the engine launches them.
"""
import math

import numpy as np
import torch

from ccinfer_b200.config import Qwen3Config
from ccinfer_b200.architectures.qwen3 import build_plan
from ccinfer_b200.engine.engine import Engine, EngineOptions, StepEntry
from ccinfer_b200.engine.runtime import Runtime
from ccinfer_b200.engine.step import GroupStep, LayerCache, StepContext
from ccinfer_b200.parts import (ChannelGatedDelta, GatedLinearAttention, GroupedQueryAttention, HeadGatedDelta,
                                LatentAttention, MixtureOfExperts, RotaryHalf, SelectiveStateSpace)

DEV = "cuda"
F64 = torch.float64
PAGE = 16
EPS = 1e-5
# width: query heads, key heads, intermediate size, vocabulary (heads of 128)
SIZES = {2048: (16, 8, 8192, 32000), 4096: (32, 8, 12288, 151936)}
HD = 128
THETA = 1000000.0


# ------------------------------------------------------------------------------------------------ cases
def listed():
    return [
        # a chat server's short turns: eight prompts of some dozen tokens in one step, then sixteen tokens each, one
        # step at a time from the CUDA graph: launches and small products
        {"name": "serve_chat", "kind": "serve", "dtype": "bfloat16", "width": 2048, "layers": 4, "requests": 8,
         "prompt": 73, "new": 16, "portion": 2048},
        # a long document read in portions of 2,048 tokens, then the first tokens of the answer
        {"name": "serve_document", "kind": "serve", "dtype": "bfloat16", "width": 4096, "layers": 4, "requests": 1,
         "prompt": 4096, "new": 12, "portion": 2048},
        # the 32-bit path, with which results are checked: two short prompts and a few tokens
        {"name": "serve_float32", "kind": "serve", "dtype": "float32", "width": 2048, "layers": 2, "requests": 2,
         "prompt": 150, "new": 3, "portion": 512},
        # the attention layer of a decode step of a busy server: 32 requests of very different lengths
        {"name": "attend_decode", "kind": "attend", "width": 4096, "requests": 32, "context": 8000},
        # latent attention: a portion of one long prompt under a window
        {"name": "latent_prompt", "kind": "latent", "width": 4096, "requests": 1, "tokens": 2048, "context": 1500,
         "window": 1024},
        # latent attention: one token each of four requests that see all they have (the smallest call)
        {"name": "latent_decode", "kind": "latent", "width": 2048, "requests": 4, "tokens": 1, "context": 3000,
         "window": 0},
        # the delta rule with a decay per channel: one prompt's portion
        {"name": "delta_prompt", "kind": "delta", "width": 4096, "requests": 1, "tokens": 2048},
        # the delta rule with a decay per head: one token each of 48 requests
        {"name": "head_delta_decode", "kind": "head_delta", "width": 4096, "requests": 48, "tokens": 1},
        # gated linear attention: portions of three prompts, of lengths that divide by nothing
        {"name": "gla_prompts", "kind": "gla", "width": 2048, "requests": 3, "tokens": 1537},
        # a state space layer: portions of two prompts
        {"name": "ssm_prompts", "kind": "ssm", "width": 4096, "requests": 2, "tokens": 2048},
        # a mixture of 32 gated experts of which a token uses 4: a portion of a prompt
        {"name": "experts_prompt", "kind": "experts", "width": 4096, "tokens": 2048},
        # the same for a decode step of eight requests: the chosen experts' weights are all that it reads
        {"name": "experts_decode", "kind": "experts", "width": 4096, "tokens": 8},
    ]


def _spread(rng, lo, hi):
    """A whole number between lo and hi, spread evenly over its logarithm."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["serve", "attend", "latent", "latent", "delta", "head_delta", "gla", "ssm", "experts", "experts"])
    width = rng.choice([2048, 4096])
    if kind == "serve":
        if rng.random() < 0.3:
            return {"kind": kind, "dtype": "float32", "width": 2048, "layers": rng.randint(1, 2),
                    "requests": rng.randint(1, 3), "prompt": _spread(rng, 5, 150), "new": rng.randint(1, 3), "portion": 512}
        requests = _spread(rng, 1, 16)
        return {"kind": kind, "dtype": "bfloat16", "width": width, "layers": rng.randint(2, 4), "requests": requests,
                "prompt": _spread(rng, 5, 4096 // requests), "new": rng.randint(1, 12),
                "portion": rng.choice([512, 2048])}
    if kind == "attend":
        return {"kind": kind, "width": width, "requests": _spread(rng, 1, 32), "context": _spread(rng, 50, 8000)}
    # single tokens of some requests, or portions of a few prompts that share a step of up to 2,048 tokens
    single = kind != "experts" and rng.random() < 0.4
    requests = _spread(rng, 1, 48) if single else _spread(rng, 1, 6)
    tokens = 1 if single else _spread(rng, 17 * requests, 2048)
    if kind == "experts":
        return {"kind": kind, "width": width, "tokens": _spread(rng, 1, 2048)}
    case = {"kind": kind, "width": width, "requests": requests, "tokens": tokens}
    if kind == "latent":
        case["window"] = rng.choice([0, 1024])
        case["context"] = _spread(rng, 20, 3000 if single else 1500)
    return case


# ------------------------------------------------------------------------------------------------ what a step brings
def _cut(total, parts, seed):
    """``total`` cut into ``parts`` uneven whole numbers, each at least 2."""
    r = np.random.RandomState(seed % (1 << 31))
    share = r.uniform(0.5, 1.5, parts)
    n = np.maximum(2, np.floor(share / share.sum() * total).astype(int))
    n[-1] = max(2, total - int(n[:-1].sum()))
    return [int(x) for x in n]


def _entries(c, seed):
    """(tokens cached before, tokens brought) of each request of the step."""
    r = np.random.RandomState((seed + 17) % (1 << 31))
    kind = c["kind"]
    if kind == "attend":
        lo = max(1, c["context"] // 16)
        return [(int(x), 1) for x in np.exp(r.uniform(math.log(lo), math.log(c["context"]), c["requests"]))]
    before = c.get("context", 0)
    if c["tokens"] == 1:
        return [(int(x), 1) for x in r.randint(max(1, before // 2), max(2, before) + 1, c["requests"])] if before \
            else [(int(x), 1) for x in r.randint(4, 3000, c["requests"])]
    counts = _cut(c["tokens"], c["requests"], seed)
    # every second prompt is one that has been read up to some place already
    return [(before if i % 2 == 0 else 0, n) for i, n in enumerate(counts)] if before else \
        [(0 if i % 2 == 0 else 512, n) for i, n in enumerate(counts)]


def _int(values):
    return torch.tensor(values, dtype=torch.int32, device=DEV)


def _step(entries, seed, paged):
    """The step as the device sees it, its pages anywhere in the pool; returns (step, slots of each request's tokens)."""
    r = np.random.RandomState((seed + 29) % (1 << 31))
    step = StepContext()
    counts = [n for _, n in entries]
    step.n_tokens, step.n_entries = sum(counts), len(entries)
    step.n_single = len(entries) if max(counts) == 1 else 0
    step.max_q_len, step.max_ctx = max(counts), max(p + n for p, n in entries)
    step.positions = _int([p + i for p, n in entries for i in range(n)])
    step.entry_of_token = _int([e for e, n in enumerate(counts) for _ in range(n)])
    step.cu_q = _int([0] + list(np.cumsum(counts)))
    step.pos0 = _int([p for p, _ in entries])
    step.ctx_after = _int([p + n for p, n in entries])
    step.state_slot = _int(list(range(len(entries))))
    slots = None
    if paged:
        pages = [-(-(p + n) // PAGE) for p, n in entries]
        total, stride = sum(pages), max(pages)
        order = r.permutation(total)
        table = np.full((len(entries), stride), -1, dtype=np.int32)
        at, slots = 0, []
        for e, k in enumerate(pages):
            table[e, :k] = order[at:at + k]
            at += k
            j = np.arange(sum(entries[e]))
            slots.append(table[e, j // PAGE].astype(np.int64) * PAGE + j % PAGE)
        new = np.concatenate([s[p:] for s, (p, _) in zip(slots, entries)]).astype(np.int32)
        step.groups = [GroupStep(index=0, page_size=PAGE, num_pages=total, window=None,
                                 slot_map=torch.from_numpy(new).to(DEV), block_table=torch.from_numpy(table).to(DEV),
                                 host_slot_map=new, host_block_table=table)]
    return step, slots


# ------------------------------------------------------------------------------------------------ weights and inputs
class _Weights:
    """Draws tensors in order: matrices bfloat16 (float32 in the 32-bit path) with rows of unit expectation, vectors
    float32."""

    def __init__(self, seed, dtype=torch.bfloat16):
        self.g = torch.Generator(device=DEV).manual_seed(int(seed))
        self.dtype, self.t = dtype, {}

    def normal(self, *shape):
        return torch.randn(shape, generator=self.g, device=DEV)

    def uniform(self, lo, hi, *shape):
        return lo + (hi - lo) * torch.rand(shape, generator=self.g, device=DEV)

    def matrix(self, name, rows, cols):
        # (the values are bfloat16 ones in both compute types, as a checkpoint's are)
        self.t[name] = (self.normal(rows, cols) * cols ** -0.5).to(torch.bfloat16).to(self.dtype)

    def matrices(self, cols, **rows):
        for name, n in rows.items():
            self.matrix(name, n, cols)

    def norm(self, name, n):
        self.t[name] = 1 + 0.1 * self.normal(n)

    def decays(self, heads, steps):
        """A rate per head between 1 and 16 and a step size between 1e-3 and 1e-1, through its inverse softplus."""
        self.t["A_log"] = torch.log(self.uniform(1.0, 16.0, heads))
        dt = torch.exp(self.uniform(math.log(1e-3), math.log(1e-1), steps))
        self.t["dt_bias"] = dt + torch.log(-torch.expm1(-dt))

    def fetch(self, name):
        return self.t[name]


def _names(*keys, **more):
    return dict({k: k for k in keys}, **more)


def _layer_weights(c, seed):
    """The tensors of the case's part, by name."""
    w = _Weights(seed)
    D = c["width"]
    H, G, F, _ = SIZES[D]
    kind = c["kind"]
    if kind == "attend":
        w.matrices(D, q=H * HD, k=G * HD, v=G * HD)
        w.matrix("o", D, H * HD)
        w.norm("q_norm", HD)
        w.norm("k_norm", HD)
    elif kind == "latent":
        w.matrices(D, q=H * HD, dkv=512 + 64, g=H)
        w.matrices(512, uk=H * 64, uv=H * HD)
        w.norm("dkv_norm", 512)
        w.t["sink"] = w.normal(H)
        w.matrix("o", D, H * HD)
    elif kind in ("delta", "head_delta"):
        w.matrices(D, q=H * HD, k=H * HD, v=H * HD, b=H)
        for n in ("q_conv", "k_conv", "v_conv"):
            w.t[n] = w.uniform(-0.5, 0.5, H * HD, 4)
        if kind == "delta":
            w.matrices(D, a1=HD, g1=HD)
            w.matrices(HD, a2=H * HD, g2=H * HD)
            w.decays(H, H * HD)
        else:
            w.matrices(D, a=H, g=H * HD)
            w.decays(H, H)
        w.norm("norm", HD)
        w.matrix("o", D, H * HD)
    elif kind == "gla":
        w.matrices(D, q=H * HD, k=H * HD, v=H * HD, g=H * HD, a1=HD)
        w.matrix("a2", H * HD, HD)
        w.t["a2_bias"] = 2 + w.normal(H * HD)
        w.norm("norm", HD)
        w.matrix("o", D, H * HD)
    elif kind == "ssm":
        heads, P, N, groups = _ssm_sizes(D)
        inner, C = heads * P, heads * P + 2 * groups * N
        w.matrix("in", inner + C + heads, D)
        w.t["conv"], w.t["conv_bias"] = w.uniform(-0.5, 0.5, C, 4), w.uniform(-0.5, 0.5, C)
        w.decays(heads, heads)
        w.norm("D", heads)
        w.norm("norm", inner)
        w.matrix("o", D, inner)
    elif kind == "experts":
        w.matrix("router", 32, D)
        for e in range(32):
            w.matrices(D, **{f"gate{e}": F // 4, f"up{e}": F // 4})
            w.matrix(f"down{e}", D, F // 4)
    return w


def _ssm_sizes(D):
    return 2 * D // 64, 64, 128, 8   # heads, channels of a head, state, groups


def _part(c):
    D = c["width"]
    H, G, F, _ = SIZES[D]
    kind = c["kind"]
    if kind == "attend":
        return GroupedQueryAttention(D, H, G, HD, RotaryHalf(HD, THETA), _names("q", "k", "v", "o", "q_norm", "k_norm"),
                                     qk_norm_eps=1e-6)
    if kind == "latent":
        return LatentAttention(D, H, 64, 64, HD, 512, c["window"] or None, HD ** -0.5, THETA, 64, EPS,
                               _names("q", "dkv", "dkv_norm", "uk", "uv", "sink", "o", "g"))
    if kind == "delta":
        return ChannelGatedDelta(D, H, H, HD, HD, 4, EPS, _names(
            "q", "k", "v", "o", "q_conv", "k_conv", "v_conv", "b", "A_log", "dt_bias", "a1", "a2", "g1", "g2", "norm",
            a_rank=HD, g_rank=HD))
    if kind == "head_delta":
        return HeadGatedDelta(D, H, H, HD, HD, 4, EPS, _names("q", "k", "v", "o", "g", "q_conv", "k_conv", "v_conv", "a",
                                                              "b", "A_log", "dt_bias", "norm"))
    if kind == "gla":
        return GatedLinearAttention(D, H, HD, HD, 16.0, HD, EPS, _names("q", "k", "v", "g", "o", "norm", "a1", "a2",
                                                                        "a2_bias"))
    if kind == "ssm":
        heads, P, N, groups = _ssm_sizes(D)
        return SelectiveStateSpace(D, heads, P, N, groups, 4, 8, EPS, _names("in", "conv", "conv_bias", "dt_bias", "A_log",
                                                                             "D", "norm", "o"))
    return MixtureOfExperts(D, 32, 4, F // 4, {"router": "router", "gate": "gate{e}", "up": "up{e}", "down": "down{e}"},
                            activation="swiglu")


def _rows(c, seed, n):
    """The part's input rows: what a norm leaves."""
    return _Weights(seed + 1).normal(n, c["width"]).to(torch.bfloat16)


def _memory(c, seed, entries):
    """The requests' states S [requests, heads, value channels, key channels]: zero for a request that begins."""
    H = SIZES[c["width"]][0]
    heads, dv, dk = (_ssm_sizes(c["width"])[0], 64, 128) if c["kind"] == "ssm" else (H, HD, HD)
    g = _Weights(seed + 2)
    S = torch.zeros((len(entries), heads, dv, dk), device=DEV)
    for e, (before, _) in enumerate(entries):
        if before:
            S[e] = 0.1 * g.normal(heads, dv, dk)
    return S


def _cached(c, seed, entries):
    """What the requests' earlier tokens left in the cache, request by request."""
    g = _Weights(seed + 3)
    G = SIZES[c["width"]][1]
    if c["kind"] == "attend":
        return [(g.normal(p, G, HD).to(torch.bfloat16), g.normal(p, G, HD).to(torch.bfloat16)) for p, _ in entries]
    return [g.normal(p, 512 + 64).to(torch.bfloat16) for p, _ in entries]


# ------------------------------------------------------------------------------------------------ prepare and run
def prepare(case, seed):
    c = case
    if c["kind"] == "serve":
        return _prepare_serve(c, seed)
    w = _layer_weights(c, seed)
    part = _part(c)
    entries = [(0, c["tokens"])] if c["kind"] == "experts" else _entries(c, seed)
    T = sum(n for _, n in entries)
    paged = c["kind"] in ("attend", "latent")
    step, slots = _step(entries, seed, paged)
    rt = Runtime(DEV + ":0", torch.bfloat16, max(T, len(entries)), len(entries))
    part.bind(rt, w.fetch)
    s = {"kind": c["kind"], "part": part, "rt": rt, "step": step, "x": _rows(c, seed, T), "cache": None, "state": None,
         "graph": None, "out": None}
    if paged:
        need, pages = part.cache_need(), step.groups[0].num_pages
        tensors = {t.name: torch.zeros((pages,) + t.page_shape(PAGE), dtype=torch.bfloat16, device=DEV)
                   for t in need.tensors}
        for old, at in zip(_cached(c, seed, entries), slots):
            page, off = (torch.from_numpy(a).to(DEV) for a in (at // PAGE, at % PAGE))
            if c["kind"] == "attend":
                n = old[0].shape[0]
                tensors["k"][page[:n], :, off[:n]] = old[0]
                tensors["v"][page[:n], :, off[:n]] = old[1]
            else:
                n = old.shape[0]
                tensors["latent"][page[:n], off[:n]] = old
        s["cache"] = LayerCache(tensors, step.groups[0], True)
    need = getattr(part, "state_need", lambda: None)()
    first = None
    if need is not None:
        first = _memory(c, seed, entries)
        if isinstance(need, (list, tuple)):
            s["state"] = {n.name: torch.zeros((len(entries),) + tuple(n.shape), dtype=n.dtype or torch.bfloat16, device=DEV)
                          for n in need}
            memory = s["state"]["S"]
        else:
            memory = s["state"] = torch.zeros_like(first)
        memory.copy_(first)
    if step.max_q_len == 1 or T <= 16:
        # a decode step: recorded once (after a run that lets every scratch buffer be there), replayed afterwards
        _forward(s)
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            s["out"] = _forward(s)
        s["graph"] = graph
        if first is not None:
            memory.copy_(first)
            for name, t in (s["state"].items() if isinstance(s["state"], dict) else ()):
                if name != "S":
                    t.zero_()
    return s


def _forward(s):
    if s["kind"] == "experts":
        return s["part"].forward(s["x"], s["step"])
    return s["part"].forward(s["x"], s["step"], s["cache"], s["state"])


def run(state):
    s = state
    if s["kind"] == "serve":
        return _run_serve(s)
    if s["graph"] is not None:
        s["graph"].replay()
        out = s["out"]
    else:
        out = _forward(s)
    if s["state"] is not None:
        return {"out": out, "state": s["state"]}
    return {"out": out}


def _prompts(c, seed):
    """Token lists: each request's prompt, and the tokens that follow it."""
    r = np.random.RandomState((seed + 41) % (1 << 31))
    V = SIZES[c["width"]][3]
    n = c["requests"]
    lens = [c["prompt"]] if n == 1 else [max(1, int(c["prompt"] * f)) for f in r.uniform(0.4, 1.0, n)]
    return [r.randint(0, V, x).tolist() for x in lens], r.randint(0, V, (c["new"], n)).tolist()


def _model_weights(c, seed):
    D = c["width"]
    H, G, F, V = SIZES[D]
    w = _Weights(seed, torch.float32 if c["dtype"] == "float32" else torch.bfloat16)
    w.matrix("model.embed_tokens.weight", V, D)
    w.t["model.embed_tokens.weight"] *= D ** 0.5   # (rows of unit size)
    for l in range(c["layers"]):
        p = f"model.layers.{l}."
        w.matrices(D, **{p + "self_attn.q_proj.weight": H * HD, p + "self_attn.k_proj.weight": G * HD,
                         p + "self_attn.v_proj.weight": G * HD, p + "mlp.gate_proj.weight": F, p + "mlp.up_proj.weight": F})
        w.matrix(p + "self_attn.o_proj.weight", D, H * HD)
        w.matrix(p + "mlp.down_proj.weight", D, F)
        for name, n in (("self_attn.q_norm", HD), ("self_attn.k_norm", HD), ("input_layernorm", D),
                        ("post_attention_layernorm", D)):
            w.norm(p + name + ".weight", n)
    w.norm("model.norm.weight", D)
    w.matrix("lm_head.weight", V, D)
    return w


def _prepare_serve(c, seed):
    D = c["width"]
    H, G, F, V = SIZES[D]
    cfg = Qwen3Config.from_json({
        "architectures": ["Qwen3ForCausalLM"], "num_hidden_layers": c["layers"], "hidden_size": D,
        "num_attention_heads": H, "num_key_value_heads": G, "head_dim": HD, "intermediate_size": F, "vocab_size": V,
        "rope_theta": THETA, "rms_norm_eps": 1e-6, "max_position_embeddings": 40960, "tie_word_embeddings": False})
    prompts, follow = _prompts(c, seed)
    held = [-(-(len(p) + c["new"]) // PAGE) * PAGE for p in prompts]
    engine = Engine(build_plan(cfg), _model_weights(c, seed).fetch, EngineOptions(
        dtype=c["dtype"], page_size=PAGE, kv_tokens=sum(held), max_requests=c["requests"],
        max_tokens_per_step=max(c["portion"], c["requests"]), max_context=max(held)))
    engine.warm_up([c["requests"]])
    logits = torch.empty((c["new"] + 1, c["requests"], V), dtype=torch.float32, device=DEV)
    return {"kind": "serve", "engine": engine, "prompts": prompts, "follow": follow, "portion": c["portion"],
            "logits": logits}


def _run_serve(s):
    """The prompts in steps of up to ``portion`` tokens, then every request's next tokens a step at a time; the logits
    after every prompt and every token."""
    engine, logits, n = s["engine"], s["logits"], len(s["prompts"])
    for i in range(n):
        engine.open_request(i)
    i, at = 0, 0
    while i < n:
        entries, rows, room = [], [], s["portion"]
        while i < n and room > 0:
            part = s["prompts"][i][at:at + room]
            room -= len(part)
            at += len(part)
            done = at == len(s["prompts"][i])
            entries.append(StepEntry(i, part, [len(part) - 1] if done else []))
            if done:
                rows.append(i)
                i, at = i + 1, 0
        got = engine.step(entries)
        if rows:
            logits[0, rows[0]:rows[-1] + 1].copy_(got)
    for k, tokens in enumerate(s["follow"]):
        logits[k + 1].copy_(engine.step([StepEntry(i, [t], [0]) for i, t in enumerate(tokens)]))
    for i in range(n):
        engine.close_request(i)
    return {"logits": logits}


# ------------------------------------------------------------------------------------------------ the same in 64 bits
def _rms(x, w=None, eps=EPS):
    y = x / torch.sqrt(x.square().mean(-1, keepdim=True) + eps)
    return y if w is None else y * w


def _turn(x, pos, freq):
    """Pairs (i, i + n) of the last axis [.., 2 n] of x [tokens, heads, 2 n] turned by pos * freq[i]."""
    a = torch.outer(pos.double(), freq)[:, None, :]
    n = freq.numel()
    u, v = x[..., :n], x[..., n:]
    return torch.cat([u * a.cos() - v * a.sin(), v * a.cos() + u * a.sin()], -1)


def _frequencies(dims):
    e = np.arange(0, dims, 2, dtype=np.float32) / np.float32(dims)
    f = np.float32(1.0) / np.power(np.float64(THETA), e.astype(np.float64)).astype(np.float32)
    return torch.from_numpy(f.astype(np.float64)).to(DEV)


def _attend(q, k, v, scale, window=0):
    """softmax(q k^T) v, causal, the queries being the last tokens: q [n, H, d], k, v [m, G, d]."""
    n, H, _ = q.shape
    m, G, _ = k.shape
    i, j = torch.arange(m - n, m, device=DEV)[:, None], torch.arange(m, device=DEV)[None]
    hidden = (j > i) | ((i - j >= window) if window else False)
    out = torch.empty((n, H, v.shape[2]), dtype=F64, device=DEV)
    for h in range(H):
        s = (q[:, h] @ k[:, h * G // H].T * scale).masked_fill_(hidden, -math.inf)
        out[:, h] = torch.softmax(s, -1) @ v[:, h * G // H]
    return out


def _conv(x, w, b=None):
    """A causal convolution over time per channel, inputs before the first row counting as zero, then silu."""
    taps = w.shape[1]
    padded = torch.cat([x.new_zeros((taps - 1, x.shape[1])), x])
    y = sum(padded[j:j + x.shape[0]] * w[:, j] for j in range(taps))
    return torch.nn.functional.silu(y if b is None else y + b)


def _recur(q, k, v, g, S, beta=None):
    """S <- g S (+ the delta rule's correction) + k v^T; o = S^T q, token by token.  q, k [T, H, dk], v [T, H, dv], g
    [T, H, dk or 1], S [H, dv, dk]; returns (o [T, H, dv], S)."""
    o = torch.empty_like(v)
    for t in range(q.shape[0]):
        S = S * g[t][:, None, :]
        u = v[t]
        if beta is not None:
            u = beta[t][:, None] * (u - (S * k[t][:, None, :]).sum(-1))
        S = S + u[:, :, None] * k[t][:, None, :]
        o[t] = (S * q[t][:, None, :]).sum(-1)
    return o, S


def exact(case, seed):
    c = case
    if c["kind"] == "serve":
        return _exact_serve(c, seed)
    w = {k: v.double() for k, v in _layer_weights(c, seed).t.items() if c["kind"] != "experts"}
    if c["kind"] == "experts":
        return _exact_experts(c, seed)
    entries = _entries(c, seed)
    x = _rows(c, seed, sum(n for _, n in entries)).double()
    H, G, _, _ = SIZES[c["width"]]
    kind = c["kind"]
    old = _cached(c, seed, entries) if kind in ("attend", "latent") else None
    memory = None if old is not None else _memory(c, seed, entries).double()
    out, at = torch.empty_like(x), 0
    for e, (before, n) in enumerate(entries):
        h = x[at:at + n]
        pos = torch.arange(before, before + n, device=DEV)
        if kind == "attend":
            q = _turn(_rms((h @ w["q"].T).view(n, H, HD), w["q_norm"], 1e-6), pos, _frequencies(HD))
            k = _turn(_rms((h @ w["k"].T).view(n, G, HD), w["k_norm"], 1e-6), pos, _frequencies(HD))
            v = (h @ w["v"].T).view(n, G, HD)
            o = _attend(q, torch.cat([old[e][0].double(), k]), torch.cat([old[e][1].double(), v]), HD ** -0.5)
        elif kind == "latent":
            o = _latent(c, w, h, pos, old[e].double(), H)
        else:
            o, memory[e] = _memories(c, w, h, memory[e], H)
        out[at:at + n] = o.reshape(n, -1) @ w["o"].T
        at += n
    if memory is None:
        return {"out": out}
    if kind == "gla":
        return {"out": out, "state": memory}
    return {"out": out, "state": {"S": memory, "conv": None}}


def _latent(c, w, h, pos, old, H):
    n = h.shape[0]
    q = (h @ w["q"].T).view(n, H, HD)
    row = h @ w["dkv"].T
    f = torch.from_numpy(np.power(THETA, -np.arange(0, 64, 2) / 64.0).astype(np.float32).astype(np.float64)).to(DEV)
    q = torch.cat([q[..., :64], _turn(q[..., 64:], pos, f)], -1)
    new = torch.cat([_rms(row[:, :512], w["dkv_norm"]), _turn(row[:, None, 512:], pos, f)[:, 0]], -1)
    rows = torch.cat([old, new])
    m = rows.shape[0]
    i, j = torch.arange(m - n, m, device=DEV)[:, None], torch.arange(m, device=DEV)[None]
    hidden = (j > i) | ((i - j >= c["window"]) if c["window"] else False)
    uk, uv = w["uk"].view(H, 64, 512), w["uv"].view(H, HD, 512)
    out = torch.empty((n, H, HD), dtype=F64, device=DEV)
    for a in range(H):
        k = torch.cat([rows[:, :512] @ uk[a].T, rows[:, 512:]], -1)
        s = (q[:, a] @ k.T * HD ** -0.5).masked_fill_(hidden, -math.inf)
        s = torch.cat([s, w["sink"][a].expand(n, 1)], -1)
        out[:, a] = torch.softmax(s, -1)[:, :m] @ (rows[:, :512] @ uv[a].T)
    return out * torch.sigmoid(h @ w["g"].T)[..., None]


def _memories(c, w, h, S, H):
    """The mixers with a state: (rows before the output projection, the state after the request's tokens)."""
    n, kind = h.shape[0], c["kind"]
    if kind == "ssm":
        heads, P, N, groups = _ssm_sizes(c["width"])
        inner, wide = heads * P, heads * P + 2 * groups * N
        z, xbc, dt = (h @ w["in"].T).split([inner, wide, heads], -1)
        xbc = _conv(xbc, w["conv"], w["conv_bias"])
        x, b, k = xbc.split([inner, groups * N, groups * N], -1)
        x = x.view(n, heads, P)
        b, k = (t.view(n, groups, N).repeat_interleave(heads // groups, 1) for t in (b, k))
        dt = torch.nn.functional.softplus(dt + w["dt_bias"])
        decay = torch.exp(-torch.exp(w["A_log"]) * dt)
        o, S = _recur(k, b, x * dt[..., None], decay[..., None], S)
        y = (o + w["D"][:, None] * x).reshape(n, inner) * torch.nn.functional.silu(z)
        return _rms(y.view(n, 8, inner // 8)).reshape(n, inner) * w["norm"], S
    q, k, v = (h @ w[t].T for t in "qkv")
    if kind == "gla":
        g = torch.sigmoid(h @ w["a1"].T @ w["a2"].T + w["a2_bias"]) ** (1 / 16.0)
        q, k, v, g = (t.view(n, H, HD) for t in (q, k, v, g))
        o, S = _recur(q * HD ** -0.5, k, v, g, S)
        gate = torch.nn.functional.silu(h @ w["g"].T)
        return (_rms(o, w["norm"]).reshape(n, -1) * gate), S
    q, k, v = (_conv(t, w[name + "_conv"]).view(n, H, HD) for t, name in ((q, "q"), (k, "k"), (v, "v")))
    q, k = (t / torch.sqrt(t.square().sum(-1, keepdim=True) + 1e-6) for t in (q, k))
    beta = torch.sigmoid(h @ w["b"].T)
    rate = torch.exp(w["A_log"])[:, None]
    if kind == "delta":
        a = (h @ w["a1"].T @ w["a2"].T + w["dt_bias"]).view(n, H, HD)
        gate = torch.sigmoid(h @ w["g1"].T @ w["g2"].T)
    else:
        a = (h @ w["a"].T + w["dt_bias"]).view(n, H, 1)
        gate = torch.nn.functional.silu(h @ w["g"].T)
    g = torch.exp(-rate * torch.nn.functional.softplus(a))
    o, S = _recur(q * HD ** -0.5, k, v, g, S, beta)
    return _rms(o, w["norm"]).reshape(n, -1) * gate, S


def _exact_experts(c, seed):
    w = _layer_weights(c, seed).t
    x = _rows(c, seed, c["tokens"]).double()
    share = torch.softmax(x @ w["router"].double().T, -1)
    best, which = share.topk(4, -1)
    out = torch.zeros_like(x)
    for e in range(32):
        rows, col = (which == e).nonzero(as_tuple=True)
        if rows.numel():
            h = x[rows]
            a = torch.nn.functional.silu(h @ w[f"gate{e}"].double().T) * (h @ w[f"up{e}"].double().T)
            out[rows] += best[rows, col][:, None] * (a @ w[f"down{e}"].double().T)
    return {"out": out}


def _exact_serve(c, seed):
    D = c["width"]
    H, G, F, V = SIZES[D]
    w = _model_weights(c, seed).t
    prompts, follow = _prompts(c, seed)
    n, new = len(prompts), c["new"]
    streams = [w["model.embed_tokens.weight"][torch.tensor(p + [follow[k][i] for k in range(new)], device=DEV)].double()
               for i, p in enumerate(prompts)]
    freq = _frequencies(HD)
    for l in range(c["layers"]):
        p = f"model.layers.{l}."
        m = {k[len(p):]: v.double() for k, v in w.items() if k.startswith(p)}
        for i, x in enumerate(streams):
            T = x.shape[0]
            pos = torch.arange(T, device=DEV)
            h = _rms(x, m["input_layernorm.weight"], 1e-6)
            q = (h @ m["self_attn.q_proj.weight"].T).view(T, H, HD)
            k = (h @ m["self_attn.k_proj.weight"].T).view(T, G, HD)
            v = (h @ m["self_attn.v_proj.weight"].T).view(T, G, HD)
            q = _turn(_rms(q, m["self_attn.q_norm.weight"], 1e-6), pos, freq)
            k = _turn(_rms(k, m["self_attn.k_norm.weight"], 1e-6), pos, freq)
            x = x + _attend(q, k, v, HD ** -0.5).reshape(T, -1) @ m["self_attn.o_proj.weight"].T
            h = _rms(x, m["post_attention_layernorm.weight"], 1e-6)
            a = torch.nn.functional.silu(h @ m["mlp.gate_proj.weight"].T) * (h @ m["mlp.up_proj.weight"].T)
            streams[i] = x + a @ m["mlp.down_proj.weight"].T
    rows = torch.stack([x[-(new + 1):] for x in streams], 1)   # [new + 1, requests, D]
    rows = _rms(rows, w["model.norm.weight"].double(), 1e-6)
    return {"logits": rows @ w["lm_head.weight"].double().T}


# ------------------------------------------------------------------------------------------------ work and tolerance
def work(case):
    """Every weight, input, cached row and state that the call must read once, what it must write, and its products."""
    c, D = case, case["width"]
    H, G, F, V = SIZES[D]
    if c["kind"] == "serve":
        size = 4 if c["dtype"] == "float32" else 2
        prompts, _ = _prompts(c, 0)
        total, steps = sum(len(p) for p in prompts), c["new"] + 1
        layer = (2 * H + 2 * G) * HD * D + 3 * F * D
        body = c["layers"] * layer
        rows = c["requests"] * steps
        reads = -(-total // c["portion"]) + c["new"]
        pairs = sum((len(p) + c["new"]) ** 2 / 2 for p in prompts)
        kv = c["layers"] * 2 * G * HD * size
        seen = sum(len(p) for p in prompts) * (c["new"] + 1)
        return {"bytes": size * (reads * body + steps * V * D) + kv * seen + 4 * rows * V + 4 * total * D,
                "flops": 2 * (total + c["requests"] * c["new"]) * body + 2 * rows * V * D
                + c["layers"] * pairs * 4 * H * HD}
    if c["kind"] == "experts":
        T = c["tokens"]
        used = 32 * (1 - (1 - 4 / 32) ** T)
        return {"bytes": 2 * (used * 3 * (F // 4) * D + 32 * D + 2 * T * D), "flops": 2 * T * (4 * 3 * (F // 4) * D + 32 * D)}
    entries = _entries(c, 0)
    T = sum(n for _, n in entries)
    if c["kind"] == "attend":
        weights = (2 * H + 2 * G) * HD * D
        keys = sum(p + n for p, n in entries)
        return {"bytes": 2 * (weights + 2 * T * D + 2 * keys * G * HD), "flops": 2 * T * weights + 4 * keys * H * HD}
    if c["kind"] == "latent":
        W = c["window"] or 1 << 30
        weights = H * HD * D + (512 + 64 + H) * D + H * (64 + HD) * 512 + H * HD * D
        pairs = sum(min(p + i + 1, W) for p, n in entries for i in range(n))
        rows = sum(min(p, W) + n for p, n in entries)
        # a query meets a cached row in the latent space: R + r coordinates for the score, R for the sum
        return {"bytes": 2 * (weights + 2 * T * D + rows * 576), "flops": 2 * T * weights + 2 * pairs * H * (576 + 512)}
    if c["kind"] == "ssm":
        heads, P, N, groups = _ssm_sizes(D)
        weights = (2 * heads * P + 2 * groups * N + heads) * D + heads * P * D
        state = heads * P * N
    else:
        weights = {"delta": 4 * H * HD * D + H * D + 2 * HD * D + 2 * H * HD * HD,
                   "head_delta": 5 * H * HD * D + 2 * H * D,
                   "gla": 5 * H * HD * D + HD * D + H * HD * HD}[c["kind"]]
        state = H * HD * HD
    per_token = {"delta": 3, "head_delta": 3, "gla": 2, "ssm": 2}[c["kind"]]   # products with the state
    return {"bytes": 2 * (weights + 2 * T * D) + 8 * state * len(entries), "flops": 2 * T * (weights + per_token * state)}


def tolerance(case):
    """About four times what the 16-bit (or 32-bit) rounding between the kernels leaves against ``exact``: 1.7e-6 for the
    32-bit path, 0.002 to 0.007 otherwise (a decay near one of gated linear attention is the most sensitive)."""
    if case["kind"] == "serve":
        return {"rel": 1e-5, "max": 1e-4} if case["dtype"] == "float32" else {"rel": 0.016, "max": 0.2}
    return {"rel": {"experts": 0.01, "gla": 0.025}.get(case["kind"], 0.016), "max": 0.2}
