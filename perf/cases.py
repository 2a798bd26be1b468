"""What a program that uses this framework has it do, as cases that can be timed and compared.

A case is a layer of one of the designs (a mixer or a feed-forward, made by `parts.make_part` and called on the rows of one
step with its share of the cache, as `Model.forward` calls it), or a whole model that replays given tokens through
`ModelRunner.step`.  Sizes are those of `bench.py`'s models at widths of 512 to 2048; spans and contexts are ragged where
serving makes them so.

A case's `spans` and `contexts` say what the requests of the step bring and have cached: items "n", "kxn" (k requests of n)
or "kxa-b" (k requests spread from a to b), separated by commas.
"""
import math

import torch

import zig_ai_b200
from zig_ai_b200 import parts
from zig_ai_b200.cache import CacheManager
from zig_ai_b200.config import config_from_dict
from zig_ai_b200.engine.batch import pack_step
from zig_ai_b200.engine.runner import ModelRunner
from zig_ai_b200.kernels import ops
from zig_ai_b200.parts.base import PartSpec

PAGE = 64
EPS = 1e-6
DEV = "cuda"


def listed():
    return [
        # one user, a short question and the first words of the answer: launches and latency count
        dict(name="generate_one", kind="generate", dtype="bfloat16", width=1024, prompts="33", new=8),
        # a small batch served at once: prompts of different lengths in one step, then decoding together
        dict(name="generate_eight", kind="generate", dtype="bfloat16", width=1024, prompts="8x96-480", new=16),
        # a portion of a long prompt: 2048 rows over what earlier portions left in the cache
        dict(name="attention_prompt", kind="attention", dtype="bfloat16", width=2048, dim=64, group=4, spans="2048", contexts="6144"),
        # a full decode batch behind contexts of thousands of positions
        dict(name="attention_singles", kind="attention", dtype="bfloat16", width=1024, dim=64, group=2, spans="64x1", contexts="64x2048-6144"),
        # the 32-bit mode, in which results are checked
        dict(name="attention_float32", kind="attention", dtype="float32", width=1024, dim=64, group=2, spans="384", contexts="128"),
        # a prompt through attention with capped scores, a bias by distance and a sink
        dict(name="shaped_prompt", kind="shaped", dtype="bfloat16", width=1024, dim=64, group=4, spans="2048", contexts="0"),
        # a prompt through attention over a shared latent
        dict(name="latent_prompt", kind="latent", dtype="bfloat16", width=1024, spans="2048", contexts="0"),
        # a prompt through the delta rule with a decay per key channel
        dict(name="delta_prompt", kind="delta", dtype="bfloat16", width=1024, dim=64, decay="channel", spans="2048", contexts="0"),
        # a mixed step of the delta rule with a decay per head: decoding requests beside odd portions, some of them continued
        dict(name="delta_mixed", kind="delta", dtype="bfloat16", width=2048, dim=64, decay="head",
             spans="8x1,777,301,64,130", contexts="8x500-3000,0,1024,0,333"),
        # a prompt through the matrix memory
        dict(name="memory_prompt", kind="memory", dtype="bfloat16", width=1024, dim=64, spans="2048", contexts="0"),
        # a prompt through the selective scan
        dict(name="scan_prompt", kind="scan", dtype="bfloat16", width=2048, spans="2048", contexts="0"),
        # a prompt through routed experts
        dict(name="experts_prompt", kind="experts", dtype="bfloat16", width=2048, spans="2048", contexts="0"),
    ]


def draw(rng):
    def log(lo, hi):
        return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 1)))))))

    kind = rng.choice(["generate", "attention", "attention", "shaped", "latent", "delta", "delta", "memory", "memory", "scan", "experts"])
    if kind == "generate":
        n = log(1, 8)
        lo = log(1, 240)
        return dict(kind=kind, dtype="bfloat16", width=rng.choice([512, 1024]), prompts="%dx%d-%d" % (n, lo, log(lo, 480)), new=rng.randint(2, 16))
    c = dict(kind=kind, dtype="bfloat16", width=rng.choice([512, 1024, 1536, 2048]))
    rows, most = log(1, 2048), 8192
    if kind in ("attention", "shaped"):
        c["group"] = rng.choice([1, 2, 4])
        c["dim"] = rng.choice([64, 64, 128])
        if kind == "attention" and rng.random() < 0.25:
            c["dtype"], c["width"], rows, most = "float32", 512 * rng.randint(1, 2), log(1, 384), 128
    elif kind in ("delta", "memory"):
        c["dim"] = rng.choice([64, 64, 128])
        if kind == "delta":
            c["decay"] = rng.choice(["channel", "head"])
    spans, contexts = [], []
    if rng.random() < 0.4:                          # decoding requests, alone or in front of the portions
        n = log(1, 64)
        lo = log(1, most)
        spans.append("%dx1" % n)
        contexts.append("%dx%d-%d" % (n, lo, log(lo, most)))
    if not spans or rng.random() < 0.5:
        for _ in range(rng.randint(1, 4)):
            spans.append("%d" % max(1, log(1, rows)))
            contexts.append("%d" % (0 if rng.random() < 0.5 else log(1, most)))
        spans[-1] = "%d" % rows
    c["spans"], c["contexts"] = ",".join(spans), ",".join(contexts)
    return c


# ------------------------------------------------------------------------------------------------ sizes
def _counts(text):
    out = []
    for item in text.split(","):
        k, _, n = item.rpartition("x")
        k = int(k) if k else 1
        a, _, b = n.partition("-")
        a, b = int(a), int(b or a)
        out += [a + (b - a) * i // max(k - 1, 1) for i in range(k)]
    return out


def _lfm2_config(width):
    return config_from_dict({
        "architectures": ["Lfm2ForCausalLM"], "model_type": "lfm2", "hidden_size": width, "num_hidden_layers": 16,
        "full_attn_idxs": [2, 5, 8, 10, 12, 14], "num_attention_heads": width // 64, "num_key_value_heads": 8, "head_dim": 64,
        "block_ff_dim": 6656 * width // 1024, "block_auto_adjust_ff_dim": True, "block_multiple_of": 256, "vocab_size": 65536,
        "rope_theta": 1000000.0, "conv_L_cache": 3, "conv_bias": False, "use_qk_norm": True, "norm_eps": 1e-5,
        "tie_embedding": True, "max_position_embeddings": 128000})


def _spec(case):
    """(family, PartSpec) of a layer case."""
    W, kind, D = case["width"], case["kind"], case.get("dim", 64)
    if kind in ("attention", "shaped"):
        H = W // D
        p = dict(hidden=W, heads=H, kv_heads=H // case["group"], head_dim=D, qk_norm=True, eps=EPS)
        if kind == "attention":
            p["position"] = PartSpec("rotary_half_split", dict(head_dim=D, theta=1000000.0))
        else:
            p.update(position=PartSpec("none", {}), scale=D ** -0.5, norm_scope="whole", q_temp=(0.1, 1024), softcap=30.0,
                     rel_bias={"rows": 32, "max": 4096}, sink=True)
        return "mixer", PartSpec("attention", p)
    if kind == "latent":
        position = PartSpec("rotary_interleaved", dict(head_dim=32, theta=10000.0, rotary_dim=32))
        return "mixer", PartSpec("latent_attention", dict(hidden=W, heads=W // 64, dim=64, rot_dim=32, vdim=64, rank=256, scale=96 ** -0.5,
                                                          eps=EPS, position=position, q_rank=384, sink=True, gate="head"))
    if kind == "delta":
        p = dict(hidden=W, heads=W // D, kv_heads=W // D // 2, dim=D, vdim=128, taps=4, eps=EPS)
        if case["decay"] == "channel":
            p.update(decay="channel", decay_rank=W // 16, gate_rank=W // 8, gate_act="sigmoid")
        return "mixer", PartSpec("gated_delta", p)
    if kind == "memory":
        return "mixer", PartSpec("mlstm", dict(hidden=W, heads=W // 128, dim=D, vdim=128, gate_cap=12.0, eps=EPS))
    if kind == "scan":
        return "mixer", PartSpec("selective_scan", dict(hidden=W, inner=2 * W, state=16, dt_rank=W // 16, taps=4))
    return "feed_forward", PartSpec("routed_experts", dict(hidden=W, ff_dim=3 * W // 2, experts=8, top=2))


def _dtype(case):
    return torch.float32 if case["dtype"] == "float32" else torch.bfloat16


# ------------------------------------------------------------------------------------------------ inputs
def _generator(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed) * 7919 + 17)


def _tensor(g, local, decl, dtype):
    """A parameter as a trained layer has it: matrices that keep a row's size, norms around one, decays spread over what a state
    remembers (a few positions up to thousands)."""
    shape = tuple(decl.shape)
    if local.endswith("a_log") or local == "ssm_a":
        t = torch.log(1.0 + 15.0 * torch.rand(shape, generator=g, device=DEV))
    elif local.endswith("dt_bias") or local == "ssm_dt.bias":
        dt = torch.exp(torch.rand(shape, generator=g, device=DEV) * math.log(100.0) + math.log(0.001))
        t = dt + torch.log(-torch.expm1(-dt))                        # softplus(t) = dt
    elif local.endswith("fgate.bias"):
        t = 3.0 + 3.0 * torch.rand(shape, generator=g, device=DEV)
    elif decl.init == "norm_weight":
        t = 0.9 + 0.2 * torch.rand(shape, generator=g, device=DEV)
    elif decl.init == "conv":
        n = shape[-1] if len(shape) == 2 else 100
        t = torch.randn(shape, generator=g, device=DEV) * (n ** -0.5 if n <= 16 else 0.1 if len(shape) == 1 else n ** -0.5)
    else:
        std = 0.02 if decl.role == "table" else (float(shape[-1]) ** -0.5 if shape else 1.0)
        if local in ("delta_a.weight", "delta_a_up.weight", "ssm_dt.weight"):
            std *= 0.5
        t = torch.randn(shape, generator=g, device=DEV) * std
    return t.to(dtype) if decl.role in ("matrix", "table") else t.float()


class _Layer:
    """The inputs of a layer case: the part, its tensors, the step's description, the cache before the step and the rows."""

    def __init__(self, case, seed):
        self.case, self.dtype = case, _dtype(case)
        family, spec = _spec(case)
        self.part = parts.make_part(family, spec)
        self.family, self.p = family, spec.params
        extra = tuple(getattr(self.part, "kernel_libs", ()))
        ops.require(self.dtype, extra)
        g = _generator(seed)
        self.tensors = {k: _tensor(g, k, d, self.dtype) for k, d in self.part.params().items()}
        self.q_lens, self.ctx = _counts(case["spans"]), _counts(case["contexts"])
        needs = parts.base.needs_of(self.part)
        pages = sum(-(-(c + n) // PAGE) for c, n in zip(self.ctx, self.q_lens))
        device = torch.device(DEV, torch.cuda.current_device())
        self.cache = CacheManager([("own", needs)], PAGE, max(pages, 1), len(self.q_lens), self.dtype, device)
        spans, rids = [], list(range(len(self.q_lens)))
        for rid, (c, n) in enumerate(zip(self.ctx, self.q_lens)):
            self.cache.admit(rid)
            self.cache.reserve(rid, c + n)
            spans.append((rid, c, [0] * n, [], self.cache.requests[rid].slot))
        self.slots = [s[4] for s in spans]
        width = max(-(-(c + n) // PAGE) for c, n in zip(self.ctx, self.q_lens))
        tables = {gi: self.cache.table_rows(rids, gi, width) for gi in self.cache.paged_groups()}
        self.tables = {gi: t.copy() for gi, t in tables.items()}
        self.step = pack_step(ops, self.dtype, device, spans, tables, pin=True)
        views = self.cache.views(0, self.step)
        need = self.part.cache_need() if hasattr(self.part, "cache_need") else None
        self.view = tuple(views) if isinstance(need, (tuple, list)) else (views[0] if views else None)
        for v in views:
            if v.pages is not None:                                   # what earlier steps left in the pages
                v.pages.normal_(generator=g)
            else:
                for slot, c in zip(self.slots, self.ctx):
                    if c > 0:
                        v.state[slot].normal_(generator=g).mul_(0.25)
                        if case["kind"] == "memory":                  # a head's running maximum, the same for every column
                            top = torch.rand((v.state.shape[1], 1), generator=g, device=DEV)
                            v.state[slot][:, -1, :] = top
        self.views = views
        self.x = torch.randn((sum(self.q_lens), case["width"]), generator=g, device=DEV).to(self.dtype)


class _Whole:
    """The inputs of a whole-model case: the tensors and the tokens of every request."""

    def __init__(self, case, seed):
        self.case, self.dtype = case, _dtype(case)
        self.cfg = _lfm2_config(case["width"])
        self.model = zig_ai_b200.build_model(self.cfg)
        g = _generator(seed)
        self.tensors = {k: _tensor(g, k.split(".", 2)[-1] if k.startswith("blk.") else k, d, self.dtype)
                        for k, d in self.model.param_decls().items()}
        self.prompts, self.new = _counts(case["prompts"]), case["new"]
        ids = torch.randint(0, self.cfg.vocab_size, (len(self.prompts), max(self.prompts) + self.new), generator=g, device=DEV).tolist()
        self.tokens = [row[:n + self.new] for row, n in zip(ids, self.prompts)]


def prepare(case, seed):
    if case["kind"] != "generate":
        layer = _Layer(case, seed)
        layer.part.bind(layer.tensors, layer.dtype)
        return layer
    w = _Whole(case, seed)
    device = torch.device(DEV, torch.cuda.current_device())
    ops.require(w.dtype, sorted({lib for p in w.model.all_parts() for lib in getattr(p, "kernel_libs", ())}))
    w.model.bind(w.tensors, w.dtype)
    longest = max(len(t) for t in w.tokens)
    cache = CacheManager(w.model.cache_needs(), PAGE, len(w.tokens) * -(-longest // PAGE), len(w.tokens), w.dtype, device)
    w.runner = ModelRunner(w.model, cache, ops, w.dtype, device)
    w.runner.enable_graphs(1024)
    w.logits = torch.empty((w.new + 1, len(w.tokens), w.cfg.vocab_size), dtype=torch.float32, device=device)
    return w


def run(state):
    if isinstance(state, _Layer):
        layer, step = state, state.step
        step.scratch.clear()
        ops.begin_forward()
        try:
            y = layer.part.forward(layer.x, step) if layer.family == "feed_forward" else layer.part.forward(layer.x, step, layer.view)
        finally:
            ops.end_forward()
        return [y] + [v.pages if v.pages is not None else v.state for v in layer.views]
    w = state
    for rid in range(len(w.tokens)):
        w.runner.add_request(rid)
    w.logits[0].copy_(w.runner.step([(rid, t[:n], [n - 1]) for rid, (t, n) in enumerate(zip(w.tokens, w.prompts))]))
    for k in range(w.new):
        w.logits[k + 1].copy_(w.runner.step([(rid, [t[n + k]], [0]) for rid, (t, n) in enumerate(zip(w.tokens, w.prompts))]))
    for rid in range(len(w.tokens)):
        w.runner.end_request(rid)
    return w.logits


# ------------------------------------------------------------------------------------------------ work and tolerance
def work(case):
    W, es = case["width"], 4 if case["dtype"] == "float32" else 2
    if case["kind"] == "generate":
        cfg, prompts, new = _lfm2_config(W), _counts(case["prompts"]), case["new"]
        kv = 512
        layer_params = 16 * 3 * W * cfg.ff_dim + 10 * 4 * W * W + 6 * (2 * W * W + 2 * kv * W)
        head, B = cfg.vocab_size * W, len(prompts)
        ctx = sum(sum(range(n, n + new)) for n in prompts)
        return {"bytes": (new + 1) * es * (layer_params + head) + ctx * 6 * 2 * kv * es + (new + 1) * B * cfg.vocab_size * 4,
                "flops": 2.0 * (sum(prompts) + B * new) * layer_params + 2.0 * B * (new + 1) * head}
    q_lens, ctx = _counts(case["spans"]), _counts(case["contexts"])
    N, S, D = sum(q_lens), len(q_lens), case.get("dim", 64)
    pairs = sum(n * c + n * (n + 1) // 2 for n, c in zip(q_lens, ctx))
    io = 2 * N * W * es
    if case["kind"] in ("attention", "shaped"):
        H = W // D
        G = H // case["group"]
        mats = 2 * W * H * D + 2 * W * G * D
        return {"bytes": io + mats * es + (sum(ctx) + N) * 2 * G * D * es, "flops": 2.0 * N * mats + 4.0 * pairs * H * D}
    if case["kind"] == "latent":
        H = W // 64
        mats = W * (384 + H + 288) + 384 * H * 96 + 2 * H * 64 * 256 + H * 64 * W
        return {"bytes": io + mats * es + (sum(ctx) + N) * 288 * es, "flops": 2.0 * N * mats + 2.0 * pairs * H * (288 + 256)}
    if case["kind"] == "delta":
        H, G = W // D, W // D // 2
        inner = W // 16 + W // 8 if case["decay"] == "channel" else H + H * 128
        mats = W * (2 * G * D + H * 128 + H + inner) + (W // 16 * H * D + W // 8 * H * 128 if case["decay"] == "channel" else 0) + H * 128 * W
        return {"bytes": io + mats * es + 8 * S * (H * D * 128 + 3 * (2 * G * D + H * 128)), "flops": 2.0 * N * mats + 8.0 * N * H * D * 128}
    if case["kind"] == "memory":
        H = W // 128
        mats = W * (2 * H * D + 2 * H * 128 + 2 * H) + H * 128 * W
        return {"bytes": io + mats * es + 8 * S * H * (D + 1) * 129, "flops": 2.0 * N * mats + 5.0 * N * H * D * 128}
    if case["kind"] == "scan":
        mats = 4 * W * W + 2 * W * (W // 16 + 32) + W // 16 * 2 * W + 2 * W * W
        return {"bytes": io + mats * es + 8 * S * 2 * W * (16 + 3), "flops": 2.0 * N * mats + 6.0 * N * 2 * W * 16}
    per = 3 * W * (3 * W // 2)
    return {"bytes": io + min(8, 2 * N) * per * es + 32 * W, "flops": 2.0 * N * 2 * per + 16.0 * N * W}


def tolerance(case):
    # 32-bit: sums of a few hundred terms in another order.  bfloat16: intermediate rows rounded to 8 bits in a few places, and
    # a whole model's rounding travels through its sixteen layers
    if case["dtype"] == "float32":
        return {"rel": 1e-5}
    return {"rel": 0.02 if case["kind"] == "generate" else 0.01}


# ------------------------------------------------------------------------------------------------ the same in 64 bits
def _rms(x, w, eps):
    y = x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps)
    return y if w is None else y * w.double()


def _rotate(x, positions, dims, theta, interleaved=False):
    """Rotate the first `dims` of the last axis of x [N, heads, D]."""
    inv = float(theta) ** (-torch.arange(0, dims, 2, dtype=torch.float64, device=x.device) / dims)
    a = positions.double()[:, None, None] * inv
    cos, sin = torch.cos(a), torch.sin(a)
    out = x.clone()
    lo, hi = (slice(0, dims, 2), slice(1, dims, 2)) if interleaved else (slice(0, dims // 2), slice(dims // 2, dims))
    out[..., lo] = x[..., lo] * cos - x[..., hi] * sin
    out[..., hi] = x[..., hi] * cos + x[..., lo] * sin
    return out


def _causal_conv(u, taps, tail, act):
    """Depthwise convolution of u [n, C] behind the last inputs `tail` [taps - 1, C]; returns (rows, new tail)."""
    L = taps.shape[1]
    full = torch.cat([tail[tail.shape[0] - (L - 1):], u]) if L > 1 else u
    y = sum(full[j:j + u.shape[0]] * taps[:, j] for j in range(L))
    return (torch.nn.functional.silu(y) if act else y), full[full.shape[0] - (L - 1):]


def _softmax_rows(s, v, sink=None):
    """softmax over the last axis (with one more term in the denominator), times v."""
    top = s.amax(-1, keepdim=True)
    if sink is not None:
        top = torch.maximum(top, sink)
    e = torch.exp(s - top)
    den = e.sum(-1, keepdim=True)
    if sink is not None:
        den = den + torch.exp(sink - top)
    return (e / den) @ v


def _exact_attention(L):
    case, t, p = L.case, {k: v.double() for k, v in L.tensors.items()}, L.p
    H, G, D, shaped = p["heads"], p["kv_heads"], p["head_dim"], case["kind"] == "shaped"
    pages, table = L.views[0].pages.double(), L.tables[0]
    x, out, at = L.x.double(), [], 0
    nm = L.part.names
    bias = None
    if shaped:
        rows, far = 32, 4096.0
        half, reach = rows // 2, max(n + c for n, c in zip(L.q_lens, L.ctx))
        n = torch.arange(max(reach, 1), dtype=torch.float64)
        bucket = torch.where(n < half, n, (half + torch.floor(torch.log(n.clamp(min=1) / half) / math.log(far / half) * (rows - half))).clamp(max=rows - 1))
        bias = t[nm["rel"]][bucket.long().to(DEV)]                                          # [distance, H]
    for s, (n, c) in enumerate(zip(L.q_lens, L.ctx)):
        pos = torch.arange(c, c + n, device=DEV)
        r = x[at:at + n]
        q, k, v = r @ t[nm["q"]].T, r @ t[nm["k"]].T, (r @ t[nm["v"]].T).view(n, G, D)
        if shaped:
            q, k = _rms(q, t[nm["q_norm"]], EPS).view(n, H, D), _rms(k, t[nm["k_norm"]], EPS).view(n, G, D)
            q = q * (1 + 0.1 * torch.log(torch.floor((pos.double() + 1) / 1024) + 1))[:, None, None]
        else:
            q, k = _rms(q.view(n, H, D), t[nm["q_norm"]], EPS), _rms(k.view(n, G, D), t[nm["k_norm"]], EPS)
            q, k = _rotate(q, pos, D, 1000000.0), _rotate(k, pos, D, 1000000.0)
        ids = torch.tensor(table[s], device=DEV).long()[:-(-(c + n) // PAGE)]
        for which, new in ((0, k), (1, v)):
            pages[ids[pos // PAGE], which, :, pos % PAGE] = new
        K, V = (pages[ids, w].transpose(0, 1).reshape(G, -1, D)[:, :c + n] for w in (0, 1))
        o = torch.empty((n, H, D), dtype=torch.float64, device=DEV)
        j = torch.arange(c + n, device=DEV)
        for h in range(H):
            for a in range(0, n, 512):
                i = pos[a:a + 512]
                sc = q[a:a + 512, h] @ K[h * G // H].T * D ** -0.5
                if shaped:
                    sc = 30.0 * torch.tanh(sc / 30.0) + bias[(i[:, None] - j).clamp(min=0), h]
                sc = sc.masked_fill(j > i[:, None], -math.inf)
                o[a:a + 512, h] = _softmax_rows(sc, V[h * G // H], t[nm["sink"]][h].view(1, 1) if shaped else None)
        out.append(o.view(n, H * D) @ t[nm["o"]].T)
        at += n
    return [torch.cat(out), pages]


def _exact_latent(L):
    t, nm, H = {k: v.double() for k, v in L.tensors.items()}, L.part.names, L.p["heads"]
    D, Dr, R = 64, 32, 256
    pages, table, x, out, at = L.views[0].pages.double(), L.tables[0], L.x.double(), [], 0
    order = torch.tensor(list(range(0, Dr, 2)) + list(range(1, Dr, 2)), device=DEV)          # the pages keep (i, i + 16) as pairs
    for s, (n, c) in enumerate(zip(L.q_lens, L.ctx)):
        pos, r = torch.arange(c, c + n, device=DEV), x[at:at + n]
        q = (_rms(r @ t[nm["dq"]].T, t[nm["dq_norm"]], EPS) @ t[nm["uq"]].T).view(n, H, D + Dr)
        d = r @ t[nm["dkv"]].T
        key = _rotate(d[:, None, R:], pos, Dr, 10000.0, True)[:, 0][:, order]
        ids = torch.tensor(table[s], device=DEV).long()[:-(-(c + n) // PAGE)]
        pages[ids[pos // PAGE], pos % PAGE] = torch.cat([_rms(d[:, :R], t[nm["dkv_norm"]], EPS), key], dim=1)
        rows = pages[ids].reshape(-1, R + Dr)[:c + n]
        qr = _rotate(q[:, :, D:], pos, Dr, 10000.0, True)[:, :, order]
        gate = torch.sigmoid(r @ t[nm["g"]].T)
        o = torch.empty((n, H, D), dtype=torch.float64, device=DEV)
        j = torch.arange(c + n, device=DEV)
        for h in range(H):
            q_lat = torch.cat([q[:, h, :D] @ t[nm["uk"]].view(H, D, R)[h], qr[:, h]], dim=1)
            for a in range(0, n, 512):
                sc = (q_lat[a:a + 512] @ rows.T * 96 ** -0.5).masked_fill(j > pos[a:a + 512, None], -math.inf)
                lat = _softmax_rows(sc, rows[:, :R], t[nm["sink"]][h].view(1, 1))
                o[a:a + 512, h] = lat @ t[nm["uv"]].view(H, D, R)[h].T * gate[a:a + 512, h, None]
        out.append(o.view(n, H * D) @ t[nm["o"]].T)
        at += n
    return [torch.cat(out), pages]


def _exact_delta(L):
    t, nm, p = {k: v.double() for k, v in L.tensors.items()}, L.part.names, L.p
    H, G, D, V, channel = p["heads"], p["kv_heads"], p["dim"], p["vdim"], L.case["decay"] == "channel"
    states, tails, x, out, at = L.views[0].state.double(), L.views[1].state.double(), L.x.double(), [], 0
    taps = torch.cat([t[nm[k]] for k in ("q_conv", "k_conv", "v_conv")])
    for s, n in enumerate(L.q_lens):
        r, slot = x[at:at + n], L.slots[s]
        u, tail = _causal_conv(torch.cat([r @ t[nm[k]].T for k in ("q", "k", "v")], dim=1), taps, tails[slot], True)
        tails[slot] = tail
        q, k, v = u[:, :G * D].view(n, G, D), u[:, G * D:2 * G * D].view(n, G, D), u[:, 2 * G * D:].view(n, H, V)
        unit = lambda a: (a * torch.rsqrt(a.square().sum(-1, keepdim=True) + 1e-6)).repeat_interleave(H // G, dim=1)
        q, k = unit(q) * D ** -0.5, unit(k)
        beta = torch.sigmoid(r @ t[nm["b"]].T)
        a = (r @ t[nm["a1"]].T) @ t[nm["a2"]].T if channel else r @ t[nm["a"]].T
        step = torch.nn.functional.softplus(a + t[nm["dt_bias"]]).view(n, H, -1)
        g = torch.exp(-torch.exp(t[nm["a_log"]])[:, None] * step)                            # [n, H, D or 1]
        S = states[slot].clone()
        o = torch.empty((n, H, V), dtype=torch.float64, device=DEV)
        for i in range(n):
            S = S * g[i][:, :, None]
            w = beta[i][:, None] * (v[i] - torch.einsum("hdv,hd->hv", S, k[i]))
            S = S + k[i][:, :, None] * w[:, None, :]
            o[i] = torch.einsum("hdv,hd->hv", S, q[i])
        states[slot] = S
        gate = (r @ t[nm["g1"]].T) @ t[nm["g2"]].T if channel else r @ t[nm["g"]].T
        gate = torch.sigmoid(gate) if channel else torch.nn.functional.silu(gate)
        out.append((_rms(o, t[nm["norm"]], EPS).reshape(n, H * V) * gate) @ t[nm["o"]].T)
        at += n
    return [torch.cat(out), states, tails]


def _exact_memory(L):
    t, nm, H, D, V = {k: v.double() for k, v in L.tensors.items()}, L.part.names, L.p["heads"], L.p["dim"], L.p["vdim"]
    states, x, out, at = L.views[0].state.double(), L.x.double(), [], 0
    for s, n in enumerate(L.q_lens):
        r = x[at:at + n]
        q, k = (r @ t[nm["q"]].T).view(n, H, D) * D ** -0.5, (r @ t[nm["k"]].T).view(n, H, D)
        v = torch.cat([(r @ t[nm["v"]].T).view(n, H, V), torch.ones((n, H, 1), dtype=torch.float64, device=DEV)], dim=2)
        gi = 12.0 * torch.tanh((r @ t[nm["i"]].T + t[nm["i_bias"]]) / 12.0)
        gf = torch.nn.functional.logsigmoid(12.0 * torch.tanh((r @ t[nm["f"]].T + t[nm["f_bias"]]) / 12.0))
        S, m = states[L.slots[s]][:, :D].clone(), states[L.slots[s]][:, D, 0].clone()
        o = torch.empty((n, H, V), dtype=torch.float64, device=DEV)
        for i in range(n):
            top = torch.maximum(gf[i] + m, gi[i])
            S = S * torch.exp(gf[i] + m - top)[:, None, None] + k[i][:, :, None] * (v[i] * torch.exp(gi[i] - top)[:, None])[:, None, :]
            m = top
            y = torch.einsum("hdv,hd->hv", S, q[i])
            o[i] = y[:, :V] / (torch.maximum(y[:, V].abs(), torch.exp(-m)) + 1e-6)[:, None]
        states[L.slots[s]][:, :D], states[L.slots[s]][:, D] = S, m[:, None]
        gate = torch.sigmoid(r @ t[nm["g"]].T)
        out.append((_rms(o, None, EPS).reshape(n, H * V) * t[nm["norm"]] * gate) @ t[nm["o"]].T)
        at += n
    return [torch.cat(out), states]


def _exact_scan(L):
    t, nm, I, R = {k: v.double() for k, v in L.tensors.items()}, L.part.names, L.p["inner"], L.p["dt_rank"]
    states, tails, x, out, at = L.views[0].state.double(), L.views[1].state.double(), L.x.double(), [], 0
    A = -torch.exp(t[nm["a_log"]])
    for s, n in enumerate(L.q_lens):
        slot = L.slots[s]
        xz = x[at:at + n] @ t[nm["in"]].T
        u, L_tail = _causal_conv(xz[:, :I], t[nm["conv"]], tails[slot], False)
        tails[slot] = L_tail
        u = torch.nn.functional.silu(u + t[nm["conv_bias"]])
        proj = u @ t[nm["x"]].T
        dt = torch.nn.functional.softplus(proj[:, :R] @ t[nm["dt"]].T + t[nm["dt_bias"]])
        B, C = proj[:, R:R + 16], proj[:, R + 16:]
        S = states[slot].clone()
        y = torch.empty((n, I), dtype=torch.float64, device=DEV)
        for i in range(n):
            S = torch.exp(dt[i][:, None] * A) * S + (dt[i] * u[i])[:, None] * B[i]
            y[i] = S @ C[i]
        states[slot] = S
        out.append(((y + t[nm["d"]] * u) * torch.nn.functional.silu(xz[:, I:])) @ t[nm["o"]].T)
        at += n
    return [torch.cat(out), states, tails]


def _exact_experts(L):
    t, nm, x = {k: v.double() for k, v in L.tensors.items()}, L.part.names, L.x.double()
    score, chosen = torch.sigmoid(x @ t[nm["router"]].T).topk(2, dim=1)
    out = torch.zeros_like(x)
    for e in range(8):
        rows, place = (chosen == e).nonzero(as_tuple=True)
        r = x[rows] * score[rows, place][:, None]
        h = torch.nn.functional.silu(r @ t[nm["gate"].format(e=e)].T) * (r @ t[nm["up"].format(e=e)].T)
        out.index_add_(0, rows, h @ t[nm["down"].format(e=e)].T)
    return [out]


def _exact_generate(w):
    cfg, t = w.cfg, {k: v.double() for k, v in w.tensors.items()}
    W, H, G, D, eps = cfg.hidden_size, cfg.num_attention_heads, 8, 64, cfg.norm_eps
    logits = torch.empty((w.new + 1, len(w.tokens), cfg.vocab_size), dtype=torch.float64, device=DEV)
    for rid, (tokens, n) in enumerate(zip(w.tokens, w.prompts)):
        h = t["token_embd.weight"][torch.tensor(tokens, device=DEV)]
        T = h.shape[0]
        pos = torch.arange(T, device=DEV)
        for i, kind in enumerate(cfg.layer_types):
            f = lambda name: t["blk.%d.%s" % (i, name)]
            x = _rms(h, f("attn_norm.weight"), eps)
            if kind == "full_attention":
                q = _rotate(_rms((x @ f("attn_q.weight").T).view(T, H, D), f("attn_q_norm.weight"), eps), pos, D, cfg.rope_theta)
                k = _rotate(_rms((x @ f("attn_k.weight").T).view(T, G, D), f("attn_k_norm.weight"), eps), pos, D, cfg.rope_theta)
                v = (x @ f("attn_v.weight").T).view(T, G, D)
                k, v = (a.repeat_interleave(H // G, dim=1).transpose(0, 1) for a in (k, v))
                s = (q.transpose(0, 1) @ k.transpose(1, 2) * D ** -0.5).masked_fill(pos > pos[:, None], -math.inf)
                h = h + _softmax_rows(s, v).transpose(0, 1).reshape(T, H * D) @ f("attn_output.weight").T
            else:
                b, c, u = (x @ f("shortconv.in_proj.weight").T).chunk(3, dim=1)
                taps = f("shortconv.conv.weight").reshape(W, -1)
                y, _ = _causal_conv(b * u, taps, torch.zeros((taps.shape[1] - 1, W), dtype=torch.float64, device=DEV), False)
                h = h + (c * y) @ f("shortconv.out_proj.weight").T
            x = _rms(h, f("ffn_norm.weight"), eps)
            h = h + (torch.nn.functional.silu(x @ f("ffn_gate.weight").T) * (x @ f("ffn_up.weight").T)) @ f("ffn_down.weight").T
        logits[:, rid] = _rms(h[n - 1:n + w.new], t["token_embd_norm.weight"], eps) @ t["token_embd.weight"].T
    return logits


def exact(case, seed):
    if case["kind"] == "generate":
        return _exact_generate(_Whole(case, seed))
    L = _Layer(case, seed)
    return {"attention": _exact_attention, "shaped": _exact_attention, "latent": _exact_latent, "delta": _exact_delta,
            "memory": _exact_memory, "scan": _exact_scan, "experts": _exact_experts}[case["kind"]](L)
