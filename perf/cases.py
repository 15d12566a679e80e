"""The engine's work as cases to time: decode steps of the whole engine, and a decoder layer's parts on the rows of a step.

Kinds of case (`"kind"`):
  decode        decode steps of a batch through `Engine.step`, one after the other (graph replay, paged cache, output head):
                the float32 logits of every step
  block         one layer of the Qwen3 decoder (norm, attention over the paged cache, norm, SwiGLU) on a step's rows
  delta         the generalised delta rule of the Kedanex decoder           gated_delta  the gated delta rule of Mifolorn
  mlstm         Mifolorn's matrix memory                                    retention    Zazulix' retention
  state_space   Gezavik's state-space mixer                                 gla          Nebanex' gated linear attention
  latent        the attention over a compressed cache of the Padodra decoder
  routed        a mixture of eight experts, two per token (Kedanex)
  swiglu        the dense feed-forward of the Qwen3 decoder

`"requests"` says which rows a step brings: "2048" is a prompt of 2,048 tokens, "1500+1" one more token of a request that has
1,500 tokens in the cache ("2040+8" in a decode case: eight steps from there), and commas stand between requests.  Layer sizes are those that `bench.py` measures (`"width"` is
the model's; heads of 64 or 128 follow from it).  A part's pass does what a step does for it: the step's integers and host-built
tables are made and uploaded, the part runs; requests with a state open before it and close after it.
"""
import math

import numpy as np
import torch

from hk_b200.cache.device import PagedCache
from hk_b200.config import config_from_dict
from hk_b200.engine import Engine, StepEntry
from hk_b200.engine.context import StepContext, bind_step, pack_step, table_parts
from hk_b200.parts import (GQAAttention, GatedDeltaRule, GatedLinearAttention, GeneralDeltaRule, LatentAttention, MLSTM, Precision,
                           PreNormBlock, RMSNorm, Retention, RotaryEmbedding, RoutedFeedForward, StateSpace, SwiGLUFeedForward)
from hk_b200.weights import random_tensors

MIXERS = ("delta", "gated_delta", "mlstm", "retention", "state_space", "gla")
EPS = 1e-6
DECODE_LAYERS = 12          # a third of the model's 36: the weights of a step stay far beyond L2
VOCAB = 151936


def listed():
    return [
        # one user's chat: a token at a time, where launches and the start of every kernel count
        {"name": "decode_1", "kind": "decode", "requests": "2040+8", "width": 4096, "dtype": "bfloat16"},
        # a loaded server's decode step
        {"name": "decode_64", "kind": "decode", "requests": ",".join(["2040+8"] * 64), "width": 4096, "dtype": "bfloat16"},
        # a whole prompt in one step
        {"name": "prompt_2048", "kind": "block", "requests": "2048", "width": 4096, "dtype": "bfloat16"},
        # the scheduler's mixed step: a portion of a prompt beside requests that decode
        {"name": "mixed_527", "kind": "block", "requests": "512+512," + ",".join(f"{c}+1" for c in range(260, 2036, 125)), "width": 4096,
         "dtype": "bfloat16"},
        # the 32-bit path, as traces are replayed: a small model's layer on a prompt of odd length
        {"name": "float32_509", "kind": "block", "requests": "509", "width": 1024, "dtype": "float32"},
        # the recurrent decoders' prompts: one long request, requests of unequal lengths, and a long one in 32-bit
        {"name": "delta_2048", "kind": "delta", "requests": "2048", "width": 4096, "dtype": "bfloat16"},
        {"name": "gated_delta_ragged", "kind": "gated_delta", "requests": "700,301,77,1", "width": 2048, "dtype": "bfloat16"},
        {"name": "mlstm_1000", "kind": "mlstm", "requests": "1000", "width": 2048, "dtype": "bfloat16"},
        {"name": "retention_2048", "kind": "retention", "requests": "2048", "width": 4096, "dtype": "bfloat16"},
        {"name": "state_space_4x512", "kind": "state_space", "requests": "512,512,512,512", "width": 2048, "dtype": "bfloat16"},
        # a prompt over the compressed cache
        {"name": "latent_2048", "kind": "latent", "requests": "2048", "width": 4096, "dtype": "bfloat16"},
        # the experts of a decode step
        {"name": "routed_64", "kind": "routed", "requests": ",".join(["0+1"] * 64), "width": 4096, "dtype": "bfloat16"},
    ]


def draw(rng):
    kind = rng.choice(["decode", "block", "block", "swiglu", "delta", "gated_delta", "mlstm", "retention", "state_space", "gla", "latent", "routed"])

    def spread(low, high):
        return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))

    def cut(total, parts):
        at = sorted(rng.sample(range(1, total), min(parts, total) - 1))
        return [b - a for a, b in zip([0] + at, at + [total])]

    case = {"kind": kind, "width": 4096 if kind == "decode" else rng.choice([2048, 4096]), "dtype": "bfloat16"}
    if kind == "decode":
        batch, context = spread(1, 64), spread(100, 2040)
        case["requests"] = ",".join(f"{max(1, int(context * rng.uniform(0.5, 1.0)))}+8" for _ in range(batch))
    elif kind in ("block", "latent"):
        rows = cut(spread(20, 2048), rng.choice([1, 1, 2, 5]))
        single = rng.choice([0, 0, 3, 20])
        case["requests"] = ",".join([f"{rng.choice([0, 0, rng.randrange(1, 900)])}+{c}" for c in rows if c > 0]
                                    + [f"{rng.randrange(1, 2040)}+1" for _ in range(single)])
        if kind == "block" and rng.random() < 0.3:
            case["dtype"], case["width"] = "float32", 1024
    elif kind in MIXERS:
        case["requests"] = ",".join(str(c) for c in cut(spread(64, 2048), rng.choice([1, 1, 2, 4, 9])))
        if rng.random() < 0.2:
            case["dtype"], case["width"] = "float32", 1024
    else:
        case["requests"] = ",".join(f"0+{c}" for c in [1] * spread(1, 300)) if rng.random() < 0.5 else str(spread(16, 2048))
    return case


def _spans(case):
    """[(tokens in the cache, new tokens)] of the case's requests."""
    out = []
    for r in case["requests"].split(","):
        cached, _, new = r.rpartition("+")
        out.append((int(cached or 0), int(new)))
    return out


def _retention_decay(heads):
    return [1.0 - 2.0 ** (-5.0 - 5.0 * h / max(heads - 1, 1)) for h in range(heads)]


def _part(case, positions):
    """The case's part of a layer, not yet bound, and the sizes that its formulas need."""
    kind, d = case["kind"], case["width"]
    h64, h128 = d // 64, d // 128
    if kind == "block":
        heads, groups = (h128, h128 // 4) if d >= 2048 else (16, 8)
        rope = RotaryEmbedding(1e6, 128, positions)
        att = GQAAttention(d, heads, groups, 128, "a.", qk_norm_eps=EPS, position=rope)
        return PreNormBlock(RMSNorm(d, EPS, "n1"), att, RMSNorm(d, EPS, "n2"), SwiGLUFeedForward(d, 3 * d, "f.")), {"H": heads, "G": groups, "hd": 128}
    if kind == "swiglu":
        return SwiGLUFeedForward(d, 3 * d, "f."), {}
    if kind == "routed":
        return RoutedFeedForward(d, d // 2, 8, 2, "f."), {"E": 8, "top": 2}
    if kind == "delta":
        return GeneralDeltaRule(d, h64, 64, "m.", norm_eps=1e-5, decay_rank=64), {"H": h64, "dk": 64, "dv": 64}
    if kind == "gated_delta":
        return GatedDeltaRule(d, h64, h128, 64, 64, 4, "m.", norm_eps=EPS), {"H": h64, "G": h128, "dk": 64, "dv": 64, "taps": 4}
    if kind == "mlstm":
        return MLSTM(d, h64, 64, 64, 15.0, "m.", norm_eps=EPS), {"H": h64, "dk": 64, "dv": 64}
    if kind == "retention":
        rope = RotaryEmbedding(5e5, 32, positions)
        return Retention(d, h64, 64, 64, _retention_decay(h64), "m.", EPS, position=rope), {"H": h64, "dk": 64, "dv": 64}
    if kind == "state_space":
        return StateSpace(d, 2 * h64, 64, 128, 8, 4, "m.", EPS, norm_groups=8), {"H": 2 * h64, "dv": 64, "N": 128, "G": 8, "taps": 4}
    if kind == "gla":
        return GatedLinearAttention(d, h128, 64, 128, 16.0, "m.", EPS, decay_rank=16), {"H": h128, "dk": 64, "dv": 128}
    if kind == "latent":
        rope = RotaryEmbedding(1e4, 64, positions)
        return LatentAttention(d, h128, 128, 64, 128, 512, "m.", EPS, 192 ** -0.5, position=rope, gate=True), \
            {"H": h128, "dn": 128, "dr": 64, "vd": 128, "r": 512}
    raise ValueError(f"no kind of case '{kind}'")


def _weights(case, seed, part, prec):
    """Random tensors as the engine draws them; biases and rates lie where trained models have them: decays that forget over
    tens to thousands of tokens, step sizes between 1/1000 and 1/10, forget gates that stand open."""
    w = random_tensors(part.param_specs(), seed, 0.02, 0.05, "cuda", dtype_of=lambda s: prec.working_dtype(s.kind))
    gen = torch.Generator("cuda").manual_seed(seed * 7 + 1)

    def uniform(name, low, high):
        w[name].copy_(torch.rand(w[name].shape, generator=gen, device="cuda") * (high - low) + low)

    kind = case["kind"]
    if kind in ("gated_delta", "state_space"):
        uniform("m.A_log", 0.0, math.log(16.0))
        uniform("m.dt_bias", math.log(1e-3), math.log(1e-1))
        w["m.dt_bias"].copy_(torch.log(torch.expm1(torch.exp(w["m.dt_bias"]))))
        for name in [n for n in w if "conv" in n and w[n].dim() == 2]:
            uniform(name, -0.5, 0.5)
    if kind == "state_space":
        w["m.D"].fill_(1.0)
    if kind == "delta":
        uniform("m.w0", -6.0, -0.5)
    if kind == "mlstm":
        uniform("m.f.b", 3.0, 6.0)
        uniform("m.i.b", -10.0, -2.0)
    if kind == "gla":
        uniform("m.a2.b", 0.0, 4.0)
    return w


def _inputs(case, seed):
    """The rows of every request, cached ones first, float32 [tokens, width]."""
    gen = torch.Generator("cuda").manual_seed(seed)
    return [torch.randn(c + n, case["width"], generator=gen, device="cuda") for c, n in _spans(case)]


def _precision(case):
    return Precision(torch.bfloat16 if case["dtype"] == "bfloat16" else torch.float32, torch.device("cuda", torch.cuda.current_device()))


class _Layer:
    """A part of a layer with its cache, the step's inputs and the requests that are in the cache."""

    def __init__(self, case, seed):
        self.case, self.spans = case, _spans(case)
        self.prec = _precision(case)
        longest = max(c + n for c, n in self.spans)
        self.part, self.sizes = _part(case, longest)
        self.weights = None
        self.part.bind(_weights(case, seed, self.part, self.prec), self.prec)
        self.tables = table_parts(self.part)
        self.keeps_state = case["kind"] in MIXERS
        specs = []
        if hasattr(self.part, "cache_specs"):
            specs = self.part.cache_specs()
        elif hasattr(self.part, "cache_spec"):
            specs = [self.part.cache_spec()]
        pages = sum(-(-(c + n) // 16) for c, n in self.spans)
        self.cache = PagedCache([specs], self.prec, 16, pages, len(self.spans), longest) if specs else None
        rows = _inputs(case, seed)
        self.slots = []
        if self.cache is not None and not self.keeps_state:
            self.slots = [self.cache.open() for _ in self.spans]
            for s, (c, n) in zip(self.slots, self.spans):
                self.cache.books.extend(s, c + n)
            self.cache.sync_tables()
            for i, (c, _) in enumerate(self.spans):
                if c:
                    self.forward(rows[i][:c].contiguous(), [(self.slots[i], 0, c)])
        elif self.cache is None:
            self.slots = list(range(len(self.spans)))
        new = torch.cat([x[c:] for x, (c, _) in zip(rows, self.spans)])
        self.x = new.contiguous() if case["kind"] == "block" else new.to(self.prec.compute).contiguous()

    def context(self, spans):
        n = sum(c for _, _, c in spans)
        slot = np.repeat([s for s, _, _ in spans], [c for _, _, c in spans])
        pos = np.concatenate([np.arange(p, p + c) for _, p, c in spans])
        counts = [c for _, _, c in spans]
        ctx = StepContext(self.prec, n, None, None, None, [s for s, _, _ in spans], np.cumsum([0] + counts[:-1]).tolist(), counts,
                          [p for _, p, _ in spans], page_tokens=16)
        packed = pack_step(np.stack([np.zeros(n), pos, slot]).astype(np.int32), ctx, self.tables)
        bind_step(ctx, packed, torch.from_numpy(packed.host).to(self.prec.device, non_blocking=True))
        return ctx

    def forward(self, x, spans):
        ctx = self.context(spans)
        kind = self.case["kind"]
        if kind == "block":
            y = x.clone()
            self.part.forward(y, ctx, self.cache.layers[0])
            return y
        y = torch.empty((x.shape[0], self.case["width"]), dtype=torch.float32, device=x.device)
        if x.dtype != self.prec.compute:
            x = x.to(self.prec.compute)
        if self.cache is None:
            self.part.forward(x, y, ctx, accumulate=False)
        else:
            caches = self.cache.layers[0]
            self.part.forward(x, y, ctx, caches if hasattr(self.part, "cache_specs") else caches[0], accumulate=False)
        return y

    def step(self):
        if self.keeps_state:
            self.slots = [self.cache.open() for _ in self.spans]
        y = self.forward(self.x, [(s, c, n) for s, (c, n) in zip(self.slots, self.spans)])
        if not self.keeps_state:
            return {"y": y}
        for s in reversed(self.slots):          # the next step's requests get the same slots
            self.cache.close(s)
        return {"y": y, **{f"state{i}": c.state for i, c in enumerate(self.cache.layers[0])}}


def _decode_shape(case):
    d = case["width"]
    return dict(architectures=["Qwen3ForCausalLM"], hidden_size=d, num_hidden_layers=DECODE_LAYERS, intermediate_size=3 * d,
                num_attention_heads=d // 128, num_key_value_heads=d // 512, head_dim=128, vocab_size=VOCAB, rope_theta=1e6,
                rms_norm_eps=EPS, tie_word_embeddings=False, max_position_embeddings=8192, initializer_range=0.02)


def _tokens(case, seed):
    rng = np.random.default_rng(seed)
    return [rng.integers(0, VOCAB, c + n).tolist() for c, n in _spans(case)]


class _Decode:
    """An engine whose requests hold their contexts; every step brings each request's next token."""

    def __init__(self, case, seed):
        self.spans, self.ids = _spans(case), _tokens(case, seed)
        self.engine = eng = Engine(config=config_from_dict(_decode_shape(case)), random_seed=seed, dtype=case["dtype"], page_tokens=16,
                                   max_tokens=sum(-(-(c + n) // 16) * 16 for c, n in self.spans), max_requests=len(self.spans),
                                   max_context=2048, max_batch_tokens=8192)
        for r, (c, _) in enumerate(self.spans):
            eng.open_request(r)
        waiting, rows = [], 0
        for r, (c, _) in enumerate(self.spans):
            if rows + c > eng.max_batch_tokens:
                eng.step(waiting)
                waiting, rows = [], 0
            waiting.append(StepEntry(r, self.ids[r][:c]))
            rows += c
        eng.step(waiting)
        self.steps = [[StepEntry(r, [ids[c + s]], [0]) for r, (ids, (c, _)) in enumerate(zip(self.ids, self.spans))]
                      for s in range(self.spans[0][1])]
        self.step()                     # the first step of a batch size captures its graph

    def step(self):
        logits = [self.engine.step(entries) for entries in self.steps]
        for r, (c, _) in enumerate(self.spans):         # back to the contexts: the next pass decodes the same tokens
            self.engine.cache.books.truncate(self.engine.slot_of(r), c)
        return {"logits": logits}


def prepare(case, seed):
    return _Decode(case, seed) if case["kind"] == "decode" else _Layer(case, seed)


def run(state):
    return state.step()


# ---- what a pass cannot do without ----------------------------------------------------------------------------------


def _attention_work(spans, heads, key, value, cache_row, element):
    """(flops, cache bytes) of an attention's scores and sums over the visible keys, every cached row once."""
    pairs = sum(n * c + n * (n + 1) // 2 for c, n in spans)
    return 2.0 * pairs * heads * (key + value), float(sum(c + 2 * n for c, n in spans) * cache_row * element)


def work(case):
    kind, d, spans = case["kind"], case["width"], _spans(case)
    el = 2 if case["dtype"] == "bfloat16" else 4
    n, R = sum(c for _, c in spans), len(spans)
    h64, h128 = d // 64, d // 128
    if kind in ("decode", "block"):
        H, G = (h128, h128 // 4) if d >= 2048 else (16, 8)
        params = d * (H + 2 * G) * 128 + H * 128 * d + 9 * d * d
        flops, cache = _attention_work(spans, H, 128, 128, 2 * G * 128, el)
        if kind == "block":
            return {"bytes": params * el + cache + n * d * 8, "flops": flops + 2.0 * n * params}
        head, steps = VOCAB * d, spans[0][1]
        cache = float(sum(steps * c + steps * (steps + 1) // 2 for c, _ in spans) * 2 * G * 128 * el)      # every step reads what is there
        return {"bytes": steps * (DECODE_LAYERS * params + head) * el + DECODE_LAYERS * cache + n * VOCAB * 4,
                "flops": DECODE_LAYERS * (flops + 2.0 * n * params) + 2.0 * n * head}
    rows = n * d * (el + 4)
    if kind == "swiglu":
        return {"bytes": 9 * d * d * el + rows, "flops": 2.0 * n * 9 * d * d}
    if kind == "routed":
        experts = min(8, 2 * n)
        return {"bytes": experts * 3 * d * (d // 2) * el + 8 * d * el + rows, "flops": 2.0 * n * (2 * 3 * d * (d // 2) + 8 * d)}
    if kind == "latent":
        H = h128
        up = H * 256 * 512
        params = d * (H * 192 + 576 + H * 128) + H * 128 * d
        # keys and values made for every visible row, or queries and sums in the latent space: whichever is less
        (made, cache), (latent, _) = _attention_work(spans, H, 192, 128, 576, el), _attention_work(spans, H, 576, 512, 576, el)
        attention = min(made + 2.0 * sum(c + m for c, m in spans) * up, latent + 2.0 * n * up)
        return {"bytes": (params + up) * el + cache + rows, "flops": attention + 2.0 * n * params}
    H, dk, dv, wide, extra = {"delta": (h64, 64, 64, 5 * d + 64, 64 * d), "gated_delta": (h64, 64, 64, 3 * d + 2 * h64, 12 * d),
                              "mlstm": (h64, 64, 64, 4 * d + 2 * h64, 0), "retention": (h64, 64, 64, 4 * d, 0),
                              "state_space": (2 * h64, 128, 64, 4 * d + 2 * 8 * 128 + 2 * h64, 4 * (2 * d + 2048)),
                              "gla": (h128, 64, 128, 3 * d + 16, 16 * (d // 2))}[kind]
    params = d * wide + H * dv * d + extra
    per_entry = {"delta": 8, "gated_delta": 7, "mlstm": 5, "retention": 5, "state_space": 5, "gla": 5}[kind]
    return {"bytes": params * el + rows + 2 * R * H * dk * dv * 4, "flops": 2.0 * n * params + float(per_entry) * n * H * dk * dv}


def tolerance(case):
    """About four times the distance from `exact` that was measured: float32 parts 0.4e-6 to 1.5e-6; one layer's part with
    bfloat16 products 1.6e-3 to 2.8e-3 (the compressed cache 3.8e-3); the logits behind twelve such layers 1.9e-2."""
    if case["dtype"] == "float32":
        return {"rel": 6e-6, "max": 1e-3}
    if case["kind"] == "decode":
        return {"rel": 8e-2, "max": 0.5}
    return {"rel": 1.5e-2 if case["kind"] == "latent" else 1e-2, "max": 0.1}


# ---- the same results in 64 bits, by the formulas alone --------------------------------------------------------------


def _rms(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _rotate(x, positions, theta, dims):
    """Dim i of the first `dims` with dim i + dims/2, by the float32 angle position * theta^(-2i/dims).  x [n, heads, dim]."""
    inv = torch.tensor([math.pow(theta, -2.0 * i / dims) for i in range(dims // 2)], dtype=torch.float64).float().cuda()
    angle = (positions.float()[:, None] * inv[None, :]).double()[:, None, :]
    a, b = x[..., :dims // 2], x[..., dims // 2:dims]
    return torch.cat([a * angle.cos() - b * angle.sin(), a * angle.sin() + b * angle.cos(), x[..., dims:]], dim=-1)


def _attend(q, k, v, scale, cached):
    """q [n, H, dk] over k [c + n, G, dk], v [c + n, G, dv], causal: [n, H, dv]."""
    n, H = q.shape[0], q.shape[1]
    rep = H // k.shape[1]
    seen = torch.arange(k.shape[0], device=q.device)[None, :] <= (cached + torch.arange(n, device=q.device))[:, None]
    out = torch.empty(n, H, v.shape[2], dtype=q.dtype, device=q.device)
    for h in range(H):
        s = (q[:, h] @ k[:, h // rep].t() * scale).masked_fill(~seen, float("-inf"))
        out[:, h] = torch.softmax(s, dim=-1) @ v[:, h // rep]
    return out


def _silu(x):
    return x * torch.sigmoid(x)


def _qwen3_layer(x, w, p, n1, n2, H, G, cached, last=None):
    """One layer on all of a request's rows (the cached ones first): the rows from `cached` on (or all) behind it."""
    names = {k: w[p["a"] + f"{k}_proj.weight"].double() for k in "qkvo"}
    T, pos = x.shape[0], torch.arange(x.shape[0], device=x.device)
    h = _rms(x, EPS) * n1
    q = _rotate(_rms((h[cached:] @ names["q"].t()).view(-1, H, 128), EPS) * w[p["a"] + "q_norm.weight"].double(), pos[cached:], 1e6, 128)
    k = _rotate(_rms((h @ names["k"].t()).view(T, G, 128), EPS) * w[p["a"] + "k_norm.weight"].double(), pos, 1e6, 128)
    v = (h @ names["v"].t()).view(T, G, 128)
    x = x[cached:] + _attend(q, k, v, 128 ** -0.5, cached).flatten(1) @ names["o"].t()
    return x + _swiglu(_rms(x, EPS) * n2, w, p["f"])


def _swiglu(h, w, p):
    g, u, dn = (w[p + f"{k}_proj.weight"].double() for k in ("gate", "up", "down"))
    return (_silu(h @ g.t()) * (h @ u.t())) @ dn.t()


def _conv(x, taps_w, bias=None):
    """The causal convolution per channel and the inputs that stay behind (oldest first)."""
    taps = taps_w.shape[1]
    padded = torch.cat([x.new_zeros(taps - 1, x.shape[1]), x])
    y = sum(padded[j:j + x.shape[0]] * taps_w[:, j] for j in range(taps))
    return _silu(y if bias is None else y + bias), padded[-(taps - 1):]


def _walk(keys, values, decay, reads, remove=None):
    """S <- decay S - remove (read^T S) + key value^T, out = S^T q, over tokens; all [n, H, .].  `remove` = (u, b): b (u^T S)."""
    n, H, dk = keys.shape
    S = keys.new_zeros(H, dk, values.shape[2])
    out = torch.empty(n, H, values.shape[2], dtype=keys.dtype, device=keys.device)
    for t in range(n):
        new = decay[t][..., None] * S
        if remove is not None:
            new = new - remove[1][t][..., None] * torch.einsum("hk,hkv->hv", remove[0][t], S)[:, None, :]
        S = new + keys[t][..., None] * values[t][:, None, :]
        out[t] = torch.einsum("hk,hkv->hv", reads[t], S)
    return out, S


def _mixer_exact(kind, x, w, z):
    """(result rows, states of one request) of a recurrent mixer on a request's rows x."""
    W = {k[2:]: v.double() for k, v in w.items()}
    n, H, dv = x.shape[0], z["H"], z["dv"]
    dk = z.get("dk", z.get("N"))
    heads = lambda t, count, size: t.view(n, count, size)       # noqa: E731
    lin = lambda name: x @ W[name].t()                           # noqa: E731
    unit = lambda t: t / torch.sqrt((t * t).sum(-1, keepdim=True) + 1e-6)   # noqa: E731
    if kind == "delta":
        r, k, v, g = heads(lin("r"), H, dk), heads(lin("k"), H, dk), heads(lin("v"), H, dv), lin("g")
        wl = torch.tanh(lin("w1")) @ W["w2"].t() + W["w0"]
        d = torch.exp(-math.exp(-0.5) * torch.sigmoid(wl)).view(n, H, dk)
        a = torch.sigmoid(lin("a") + W["a.b"]).view(n, H, dk)
        u = unit(k)
        o, S = _walk(k, v, d, r, (u, a * u))
        y = _rms(o, 1e-5).flatten(1) * W["norm"] * torch.sigmoid(g)
        return y @ W["o"].t(), [S]
    if kind == "gated_delta":
        G = z["G"]
        raw = torch.cat([lin("q"), lin("k"), lin("v")], dim=1)
        act, tail = _conv(raw, torch.cat([W["q.conv"], W["k.conv"], W["v.conv"]]))
        q, k, v = act[:, :G * dk], act[:, G * dk:2 * G * dk], act[:, 2 * G * dk:]
        rep = lambda t: unit(heads(t, G, dk)).repeat_interleave(H // G, dim=1)   # noqa: E731
        q, k, v = rep(q) * dk ** -0.5, rep(k), heads(v, H, dv)
        beta = torch.sigmoid(lin("b"))
        g = torch.exp(-torch.exp(W["A_log"]) * torch.nn.functional.softplus(lin("a") + W["dt_bias"]))
        gk = g[..., None].expand(n, H, dk)
        o, S = _walk(k * beta[..., None], v, gk, q, (k * (g * beta)[..., None], k))
        y = (_rms(o, EPS) * W["norm"]).flatten(1) * _silu(lin("g"))
        return y @ W["o"].t(), [S, tail]
    if kind == "mlstm":
        q, k, v = heads(lin("q"), H, dk) * dk ** -0.5, heads(lin("k"), H, dk), heads(lin("v"), H, dv)
        cap = lambda t: 15.0 * torch.tanh(t / 15.0)              # noqa: E731
        i, f = cap(lin("i") + W["i.b"]), torch.nn.functional.logsigmoid(cap(lin("f") + W["f.b"]))
        m, ms, mbefore = x.new_zeros(H), [], []
        for t in range(n):
            mbefore.append(m)
            m = torch.maximum(f[t] + m, i[t])
            ms.append(m)
        M, B = torch.stack(ms), torch.stack(mbefore)
        keep, put = torch.exp(f + B - M), torch.exp(i - M)
        v1 = torch.cat([v, v.new_ones(n, H, 1)], dim=2)
        o, S = _walk(k * put[..., None], v1, keep[..., None].expand(n, H, dk), q)
        num, den = o[..., :dv], torch.maximum(o[..., dv:].abs(), torch.exp(-M)[..., None]) + 1e-6
        y = _rms(num / den, EPS).flatten(1) * W["norm"] * torch.sigmoid(lin("g"))
        pad = ((dv + 4) & ~3) - dv - 1
        return y @ W["o"].t(), [torch.cat([S, S.new_zeros(H, dk, pad)], dim=2), m]
    if kind == "retention":
        pos = torch.arange(n, device=x.device)
        q, k = (_rotate(heads(lin(c), H, dk), pos, 5e5, 32) for c in "qk")
        decay = torch.tensor(_retention_decay(H), dtype=torch.float64).float().double().cuda()[None, :, None].expand(n, H, dk)
        o, S = _walk(k * dk ** -0.5, heads(lin("v"), H, dv), decay, q)
        return (_rms(o, EPS).flatten(1) * _silu(lin("g"))) @ W["o"].t(), [S]
    if kind == "state_space":
        I, G, N = H * dv, z["G"], z["N"]
        p = lin("in")
        gate, raw, dt = p[:, :I], p[:, I:2 * I + 2 * G * N], p[:, 2 * I + 2 * G * N:]
        act, tail = _conv(raw, W["conv"], W["conv.b"])
        xs = heads(act[:, :I], H, dv)
        B, C = (act[:, I + j * G * N:I + (j + 1) * G * N].view(n, G, N).repeat_interleave(H // G, dim=1) for j in (0, 1))
        dt = torch.nn.functional.softplus(dt + W["dt_bias"])
        o, S = _walk(B * dt[..., None], xs, torch.exp(-torch.exp(W["A_log"]) * dt)[..., None].expand(n, H, N), C)
        y = (o + W["D"][None, :, None] * xs).flatten(1) * _silu(gate)
        return (_rms(y.view(n, 8, I // 8), EPS).flatten(1) * W["norm"]) @ W["o"].t(), [S.transpose(1, 2), tail]
    q, k, v = heads(lin("q"), H, dk) * dk ** -0.5, heads(lin("k"), H, dk), heads(lin("v"), H, dv)
    alpha = torch.exp(torch.nn.functional.logsigmoid(lin("a1") @ W["a2"].t() + W["a2.b"]) / 16.0).view(n, H, dk)
    o, S = _walk(k, v, alpha, q)
    return ((_rms(o, EPS) * W["norm"]).flatten(1) * _silu(lin("g"))) @ W["o"].t(), [S.transpose(1, 2)]


def _latent_exact(x, w, z, cached):
    H, dn, dr, vd, r = z["H"], z["dn"], z["dr"], z["vd"], z["r"]
    W = {k[2:]: v.double() for k, v in w.items()}
    T, pos = x.shape[0], torch.arange(x.shape[0], device=x.device)
    q = (x[cached:] @ W["q"].t()).view(-1, H, dn + dr)
    row = x @ W["dkv"].t()
    c = _rms(row[:, :r], EPS) * W["dkv.norm"]
    kr = _rotate(row[:, None, r:], pos, 1e4, dr)
    qr = _rotate(q[..., dn:], pos[cached:], 1e4, dr)
    ql = torch.einsum("nhd,hdr->nhr", q[..., :dn], W["uk"].view(H, dn, r))
    lat = _attend(torch.cat([ql, qr], dim=-1), torch.cat([c[:, None], kr], dim=-1), c[:, None], 192 ** -0.5, cached)
    o = torch.einsum("nhr,hvr->nhv", lat, W["uv"].view(H, vd, r)).flatten(1)
    return (o * torch.sigmoid(x[cached:] @ W["g"].t())) @ W["o"].t()


def _routed_exact(x, w, z):
    W = {k[2:]: v.double() for k, v in w.items()}
    best, ids = (x @ W["router"].t()).topk(z["top"], dim=1)
    p = torch.softmax(best, dim=1)
    y = torch.zeros_like(x)
    for e in range(z["E"]):
        row, col = torch.nonzero(ids == e, as_tuple=True)
        if row.numel():
            h = x[row]
            y.index_add_(0, row, p[row, col, None] * ((_silu(h @ W[f"e{e}.gate"].t()) * (h @ W[f"e{e}.up"].t())) @ W[f"e{e}.down"].t()))
    return y


@torch.no_grad()
def exact(case, seed):
    kind, spans, prec = case["kind"], _spans(case), _precision(case)
    if kind == "decode":
        if sum(c + n for c, n in spans) > 8192:
            return None
        from hk_b200.config import resolve_architecture
        cfg = config_from_dict(_decode_shape(case))
        specs = resolve_architecture(cfg.architecture)[1](cfg, 2048).param_specs()
        w = random_tensors(specs, seed, 0.02, 0.05, "cuda", dtype_of=lambda s: prec.working_dtype(s.kind))
        H, G, out = case["width"] // 128, case["width"] // 512, []
        for ids, (c, _) in zip(_tokens(case, seed), spans):
            x = w["model.embed_tokens.weight"][torch.tensor(ids, device="cuda")].double()
            for i in range(DECODE_LAYERS):
                p = f"model.layers.{i}."
                last = c if i == DECODE_LAYERS - 1 else 0
                x = _qwen3_layer(x, w, {"a": p + "self_attn.", "f": p + "mlp."}, w[p + "input_layernorm.weight"].double(),
                                 w[p + "post_attention_layernorm.weight"].double(), H, G, last)
            out.append(_rms(x, EPS) * w["model.norm.weight"].double())
        h, head = torch.stack(out, dim=1), w["lm_head.weight"]              # [steps, requests, width]
        return {"logits": list(torch.cat([h @ head[i:i + 16384].double().t() for i in range(0, VOCAB, 16384)], dim=2))}
    part, z = _part(case, max(c + n for c, n in spans))
    w = _weights(case, seed, part, prec)
    rows = _inputs(case, seed)
    if kind == "block":
        w["n1"], w["n2"] = w["n1"].double(), w["n2"].double()
        return {"y": torch.cat([_qwen3_layer(x.double(), w, {"a": "a.", "f": "f."}, w["n1"], w["n2"], z["H"], z["G"], c)
                                for x, (c, _) in zip(rows, spans)])}
    rows = [x.to(prec.compute).double() for x in rows]
    if kind == "latent":
        return {"y": torch.cat([_latent_exact(x, w, z, c) for x, (c, _) in zip(rows, spans)])}
    if kind == "routed":
        return {"y": _routed_exact(torch.cat(rows), w, z)}
    if kind == "swiglu":
        return {"y": _swiglu(torch.cat(rows), w, "f.")}
    if sum(n for _, n in spans) * len(spans) > 40000:
        return None
    got = [_mixer_exact(kind, x, w, z) for x in rows]
    out = {"y": torch.cat([y for y, _ in got])}
    for i in range(len(got[0][1])):
        full = torch.zeros((len(spans),) + tuple(got[0][1][i].shape), dtype=torch.float64, device="cuda")
        for slot, (_, states) in enumerate(got):        # a new cache hands its slots out in order
            full[slot] = states[i]
        out[f"state{i}"] = full
    return out

