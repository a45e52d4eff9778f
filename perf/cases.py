"""The work whose speed matters: passes of the whole-iteration executors that serve requests on one GPU.

Every case is one pass over a batch of sequences, each with ``past`` tokens in the cache and ``new`` ones in the pass:

  decode   one new token for every running sequence, replayed from the captured graph of the batch size
  prefill  whole prompts packed together, as they are admitted
  mixed    one decode token for every running sequence beside portions of prompts, the first of which goes on with a prompt
           that earlier passes began (chunked prefill)

The models are the presets with fewer of their equal layers (every kind of layer of a design is there), bf16, random weights.
MoE decoders meet random keys and values as history; layer-list decoders one that they computed themselves. A pass returns
the logits of the sampled rows and the caches and states it updated.
"""
import math
import re

import torch

from disagmoe_b200.config import (AttentionSpec, CacheConfig, ChannelDeltaSpec, GatedLinearSpec, GatedUnitSpec, HeadDecaySpec,
                                  LatentAttentionSpec, LayerListConfig, MatrixMemorySpec, SideBySideSpec, WkvSpec, get_preset)
from disagmoe_b200.models import weights as W
from disagmoe_b200.models.registry import make_executor

BLOCK = 16
#: Layers taken from the front of a preset.
LAYERS = {"mixtral": 2, "qwen-moe": 3, "deepseek-v2-lite": 3, "rurunex": 6, "supinex": 4, "vufinex": 4, "panarax": 3}
MOE = ("mixtral", "qwen-moe", "deepseek-v2-lite")


# ---- cases -------------------------------------------------------------------------------------------------------------------
def listed():
    decode = lambda name, model, batch, lo, hi: dict(name=name, model=model, phase="decode", batch=batch, ctx_min=lo, ctx_max=hi)
    prefill = lambda name, model, tokens, prompts: dict(name=name, model=model, phase="prefill", tokens=tokens, prompts=prompts)
    return [
        # one user alone on the server: every launch counts
        decode("mixtral-decode-1", "mixtral", 1, 300, 300),
        # the headline benchmark's running batch at its context lengths
        decode("mixtral-decode-256", "mixtral", 256, 192, 1536),
        # an ordinary batch of an odd size with long histories: a key / value head per query head
        decode("qwen-moe-decode-37", "qwen-moe", 37, 500, 4000),
        # small experts, many of them, a dense first layer
        decode("deepseek-v2-lite-decode-96", "deepseek-v2-lite", 96, 100, 2000),
        # a full admission pass: as many prompt tokens as the engine packs by default
        prefill("mixtral-prefill-4096", "mixtral", 4096, 3),
        # a few short prompts of ragged lengths
        prefill("deepseek-v2-lite-prefill-1111", "deepseek-v2-lite", 1111, 5),
        # the mixed engine's step at its default prompt budget
        dict(name="qwen-moe-mixed-64-512", model="qwen-moe", phase="mixed", batch=64, ctx_min=100, ctx_max=1500, tokens=512, prompts=2),
        # one long prompt through two kinds of recurrence and windowed attention
        prefill("rurunex-prefill-4096", "rurunex", 4096, 1),
        # attention with sinks and windowed latent attention, experts beside them
        prefill("supinex-prefill-3000", "supinex", 3000, 2),
        # time mixing, gated latent attention, chunked attention and grouped sigmoid routers in a mixed step
        dict(name="vufinex-mixed-24-700", model="vufinex", phase="mixed", batch=24, ctx_min=50, ctx_max=900, tokens=700, prompts=1),
        # attention beside a matrix memory, diagonal recurrence, lightning attention: prompts and decoding
        prefill("panarax-prefill-2500", "panarax", 2500, 4),
        decode("panarax-decode-48", "panarax", 48, 50, 500),
    ]


def draw(rng):
    spread = lambda lo, hi: int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    model, phase = rng.choice(list(LAYERS)), rng.choice(("decode", "prefill", "mixed"))
    case = dict(model=model, phase=phase)
    if phase != "prefill":
        # histories of layer-list decoders are computed before the pass: at most 24,000 tokens of them
        batch = spread(1, 256 if model in MOE else 64)
        top = spread(64, 4000 if model in MOE else max(64, min(2000, 24000 // batch)))
        while batch * top > 300000:
            top //= 2
        case.update(batch=batch, ctx_min=rng.randint(1, top), ctx_max=top)
    if phase != "decode":
        tokens = spread(16, 4000 if phase == "prefill" else 1000)
        case.update(tokens=tokens, prompts=rng.randint(1, max(1, min(6, tokens // 16))))
    return case


def sequences(case):
    """(past, new) tokens of every sequence of a pass, decode rows first."""
    out = []
    if case["phase"] != "prefill":
        n, lo, hi = case["batch"], case["ctx_min"], case["ctx_max"]
        # evenly spread contexts in an order that has nothing to do with their lengths
        out += [(lo + (hi - lo) * (i * 7919 % n) // max(1, n - 1), 1) for i in range(n)]
    if case["phase"] != "decode":
        n, left = case["prompts"], case["tokens"]
        for i in range(n):
            # ragged shares: each prompt takes from 1 / 2 to all of an equal share of what is left, the last the rest
            new = left if i == n - 1 else max(1, left // (n - i) * (7 + i * 5 % 7) // 14)
            out.append((300 if case["phase"] == "mixed" and i == 0 else 0, new))
            left -= new
    return out


def config(case, seed=0):
    cfg, n = get_preset(case["model"]), LAYERS[case["model"]]
    extra = dict(layers=cfg.layers[:n]) if isinstance(cfg, LayerListConfig) else {}
    return cfg.clone(num_layers=n, seed=seed, **extra)


# ---- inputs ------------------------------------------------------------------------------------------------------------------
def weights(cfg):
    """Random weights. What a sublayer adds to the residual stream is small beside the stream, as at the usual initialisation
    (output maps of 32-layer MoE decoders scaled by 1 / sqrt(2 x 32)) and in trained models. Sandwich blocks need no such
    scale: they norm what they add."""
    sd = W.init_state_dict(cfg, "cuda", cfg.dtype)
    layer_list = isinstance(cfg, LayerListConfig)
    if layer_list and cfg.block == "sandwich":
        return sd
    for n, t in sd.items():
        if n in ("embed_tokens.weight", "embed", "pos"):
            t.mul_(50.0 / (cfg.embed_scale if layer_list and n == "embed" else 1.0))
        elif re.search(r"o_proj.weight$|w2_weight$|\.o$|\.down$", n):
            t.mul_(0.125)
    return sd


def tokens_of(cfg, seed, i, n):
    """The first n tokens of sequence i."""
    return torch.randint(0, cfg.vocab_size, (n,), generator=torch.Generator().manual_seed(seed * 4099 + i), dtype=torch.int32)


def pages(seqs, seed):
    """Pages of every sequence, scattered over the pool as after some time of serving; and how many the pool has."""
    need = [(past + new + BLOCK - 1) // BLOCK for past, new in seqs]
    order = torch.randperm(sum(need), generator=torch.Generator().manual_seed(seed)).tolist()
    out, at = [], 0
    for n in need:
        out.append(order[at:at + n])
        at += n
    return out, sum(need)


def rows(parts, where):
    """Pinned host inputs of a pass: parts = (sequence, its token ids, position of the first)."""
    pos = torch.cat([torch.arange(p, p + len(ids)) for _, ids, p in parts])
    row = torch.cat([torch.full((len(ids),), i) for i, ids, _ in parts])
    slots = torch.cat([torch.tensor(where[i])[p // BLOCK] * BLOCK + p % BLOCK
                       for (i, ids, first) in parts for p in [torch.arange(first, first + len(ids))]])
    ids = torch.cat([ids for _, ids, _ in parts])
    return [t.contiguous().pin_memory() for t in (ids.int(), pos.int(), slots.long(), (pos + 1).int(), row.int())]


def history(cfg, seed, shape):
    return torch.empty(shape, dtype=cfg.dtype, device="cuda").normal_(0.0, 1.0, generator=torch.Generator("cuda").manual_seed(seed))


def prepare(case, seed):
    cfg, seqs = config(case, seed), sequences(case)
    where, n_pages = pages(seqs, seed)
    decode, total = case["phase"] == "decode", sum(new for _, new in seqs)
    past_rows = 0 if case["model"] in MOE else max((past for past, _ in seqs), default=0)
    cap = max(total, len(seqs) + 1, min(4096, sum(past for past, _ in seqs)) if past_rows else 0, past_rows)
    ex = make_executor(cfg, CacheConfig(block_size=BLOCK), device="cuda", max_batch_size=len(seqs), max_prefill_tokens=cap,
                       state_dict=weights(cfg), num_blocks=n_pages)
    for i, blocks in enumerate(where):
        ex.set_block_table_row(i, blocks)
    if decode:
        ex.capture([len(seqs)])
    ids = [tokens_of(cfg, seed, i, past + new) for i, (past, new) in enumerate(seqs)]
    if case["model"] in MOE:
        ex.kv_cache.copy_(history(cfg, seed, ex.kv_cache.shape))
        caches = [ex.kv_cache]
    else:
        caches = [t for i in sorted(ex.kv) for t in ex.kv[i]] + [t for i in sorted(ex.states) for t in ex.states[i].tensors()]
        for t in caches:
            t.zero_()
        batch = []
        for i, (past, _) in enumerate(seqs):
            if batch and sum(len(x) for _, x, _ in batch) + past > cap:
                ex.prefill(*rows(batch, where), out_rows=[0])
                batch = []
            if past:
                batch.append((i, ids[i][:past], 0))
        if batch:
            ex.prefill(*rows(batch, where), out_rows=[0])
    args = rows([(i, ids[i][past:], past) for i, (past, _) in enumerate(seqs)], where)
    ends, at = [], -1
    for _, new in seqs:
        at += new
        ends.append(at)
    torch.cuda.synchronize()
    return dict(ex=ex, args=args, ends=ends, decode=decode, caches=caches)


def run(state):
    ex = state["ex"]
    if state["decode"]:
        _, logits = ex.decode(*state["args"], want_logits=True)
    else:
        _, logits = ex.prefill(*state["args"], want_logits=True, out_rows=state["ends"])
    return dict(logits=logits, caches=state["caches"])


# ---- what a pass cannot do without -----------------------------------------------------------------------------------------------
def work(case):
    cfg, seqs = config(case), sequences(case)
    T, n = sum(new for _, new in seqs), len(seqs)
    visible = lambda window: [(min(past + new, window + new) if window else past + new) for past, new in seqs]
    pairs = lambda window: sum(sum(min(p + 1, window) if window else p + 1 for p in range(past, past + new)) for past, new in seqs)
    size = 2
    read = flops = 0
    hit = lambda experts, top: experts * (1.0 - (1.0 - top / experts) ** T)
    for name, shape in W.param_shapes(cfg).items():
        count = math.prod(shape)
        if name in ("embed_tokens.weight", "embed", "pos"):
            read += min(T, shape[0]) * shape[1] * size
            if not (name == "embed" and cfg.tied_head):
                continue
        layer = re.match(r"l(\d+)\.mlp\.e\d+\.", name)
        if layer:
            r = cfg.layers[int(layer.group(1))].routed
            read += count * size * hit(r.experts, r.top) / r.experts
            flops += 2 * count * T * r.top / r.experts
        elif ".experts." in name:
            read += count * size * hit(cfg.num_experts, cfg.top_k) / cfg.num_experts
            flops += 2 * count * T * cfg.top_k / cfg.num_experts
        elif len(shape) >= 2:
            read += count * size
            flops += 2 * count * (n if name in ("lm_head.weight", "head", "embed") else T)

    def attention(heads, dim, vdim, cached, window):
        """cached: numbers kept per token."""
        return size * cached * (sum(visible(window)) + T), 2 * heads * (dim + vdim) * pairs(window)

    def mixer(m):
        if isinstance(m, SideBySideSpec):
            return [sum(x) for x in zip(mixer(m.left), mixer(m.right))]
        if isinstance(m, LatentAttentionSpec):
            return attention(m.heads, m.dim + m.rot_dim, m.vdim, m.kv_rank + m.rot_dim, m.window)
        if isinstance(m, AttentionSpec):
            return attention(m.heads, m.dim, m.vdim, m.kv_heads * (m.dim + m.vdim), m.window or m.chunk)
        if isinstance(m, GatedUnitSpec):
            return 2 * n * m.width * 4, 8 * T * m.width
        return 2 * n * m.heads * m.dim * m.vdim * 4, 4 * T * m.heads * m.dim * m.vdim
    if isinstance(cfg, LayerListConfig):
        parts = [mixer(layer.mixer) for layer in cfg.layers]
    else:
        parts = [attention(cfg.num_heads, cfg.head_dim, cfg.head_dim, 2 * cfg.num_kv_heads * cfg.head_dim, None)] * cfg.num_layers
    return {"bytes": read + sum(b for b, _ in parts) + 4 * n * cfg.vocab_size, "flops": flops + sum(f for _, f in parts)}


def tolerance(case):
    """bf16 activations and caches. Two correct passes choose another expert for a row whose scores are nearly equal, so single
    rows differ by more than the rest."""
    return {"rel": 0.02, "max": 0.5}


# ---- the same in 64 bits, in plain torch -------------------------------------------------------------------------------------------
def exact(case, seed):
    cfg, seqs = config(case, seed), sequences(case)
    layer_list = isinstance(cfg, LayerListConfig)
    if layer_list and sum(past + new for past, new in seqs) > 20000:
        return None
    where, n_pages = pages(seqs, seed)
    sd = weights(cfg)
    ids = [tokens_of(cfg, seed, i, past + new).long().cuda() for i, (past, new) in enumerate(seqs)]
    with torch.no_grad():
        if layer_list:
            return dict(logits=layer_list_logits(cfg, sd, ids), caches=None)
        return moe_pass(cfg, sd, seqs, ids, where, n_pages, seed)


def rms(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def softplus(x):
    return x.clamp(min=0) + torch.log1p(torch.exp(-x.abs()))


def silu(x):
    return x * torch.sigmoid(x)


def gelu_tanh(x):
    return 0.5 * x * (1.0 + torch.tanh(math.sqrt(2.0 / math.pi) * (x + 0.044715 * x ** 3)))


def turn(x, pos, freqs, mult=1.0, interleaved=False):
    """Rotates pairs of the first 2 len(freqs) numbers of every head; x [T, heads, dim]."""
    a = pos.double()[:, None, None] * torch.tensor(freqs, dtype=torch.float64, device=x.device)
    c, s, n = torch.cos(a) * mult, torch.sin(a) * mult, len(freqs)
    u, v = (x[..., 0:2 * n:2], x[..., 1:2 * n:2]) if interleaved else (x[..., :n], x[..., n:2 * n])
    p, q = u * c - v * s, v * c + u * s
    both = torch.stack([p, q], -1).flatten(-2) if interleaved else torch.cat([p, q], -1)
    return torch.cat([both, x[..., 2 * n:]], -1)


def rotate(x, pos, rot):
    if rot is None:
        return x
    freqs, mult = [rot.base ** (-2.0 * i / rot.dims) for i in range(rot.dims // 2)], 1.0
    if rot.factor is not None:
        at = lambda turns: rot.dims * math.log(rot.original / (2 * math.pi * turns)) / (2 * math.log(rot.base))
        lo, hi = max(math.floor(at(rot.fast)), 0), min(math.ceil(at(rot.slow)), rot.dims - 1)
        ramp = [min(max((i - lo) / max(hi - lo, 0.001), 0.0), 1.0) for i in range(rot.dims // 2)]
        freqs = [f / rot.factor * r + f * (1 - r) for f, r in zip(freqs, ramp)]
        mult = 0.1 * math.log(rot.factor) + 1.0
    return turn(x, pos, freqs, mult, rot.interleaved)


def attend(q, k, v, scale, pos, window=None, chunk=None, softcap=None, sink=None):
    """q [T, H, D] at positions pos, k [S, G, D], v [S, G, V] from position 0 -> [T, H * V]."""
    T, H = q.shape[:2]
    keys = torch.arange(k.shape[0], device=q.device)
    hidden = keys[None] > pos[:, None]
    if window:
        hidden |= keys[None] <= pos[:, None] - window
    if chunk:
        hidden |= keys[None] < pos[:, None] // chunk * chunk
    out = []
    for h in range(H):
        g = h * k.shape[1] // H
        s = (q[:, h] @ k[:, g].T) * scale
        if softcap:
            s = softcap * torch.tanh(s / softcap)
        s = s.masked_fill(hidden, -math.inf)
        if sink is not None:
            s = torch.cat([s, sink[h].expand(T, 1)], 1)
        out.append(torch.softmax(s, -1)[:, :k.shape[0]] @ v[:, g])
    return torch.cat(out, -1)


def gated(h, w13, w2):
    """w13 [H, 2 I], w2 [I, H]."""
    y = h @ w13.double()
    n = y.shape[1] // 2
    return (silu(y[:, :n]) * y[:, n:]) @ w2.double()


def moe_pass(cfg, sd, seqs, ids, where, n_pages, seed):
    new = [n for _, n in seqs]
    pos = [torch.arange(p, p + n, device="cuda") for p, n in seqs]
    slots = [torch.tensor(b, device="cuda").repeat_interleave(BLOCK) * BLOCK + torch.arange(BLOCK, device="cuda").repeat(len(b)) for b in where]
    hd, H, G = cfg.head_dim, cfg.num_heads, cfg.num_kv_heads
    kv = history(cfg, seed, (cfg.num_layers, 2, n_pages, BLOCK, G, hd)).double()
    freqs = [cfg.rope_theta ** (-2.0 * i / hd) for i in range(hd // 2)]
    x = sd["embed_tokens.weight"][torch.cat([t[p:] for t, (p, _) in zip(ids, seqs)])].double()
    norm = lambda x, name: rms(x, cfg.rms_norm_eps) * sd[name].double()
    for l in range(cfg.num_layers):
        p, K, V = f"layers.{l}.", kv[l, 0].view(-1, G, hd), kv[l, 1].view(-1, G, hd)
        qkv = (norm(x, p + "pre_attention_layernorm.weight") @ sd[p + "qkv_proj.weight"].double().T).split(new)
        out = []
        for y, at, s, (past, n) in zip(qkv, pos, slots, seqs):
            y = y.view(n, H + 2 * G, hd)
            K[s[past:past + n]], V[s[past:past + n]] = turn(y[:, H:H + G], at, freqs), y[:, H + G:]
            out.append(attend(turn(y[:, :H], at, freqs), K[s[:past + n]], V[s[:past + n]], hd ** -0.5, at))
        x = x + torch.cat(out) @ sd[p + "o_proj.weight"].double().T
        h = norm(x, p + "post_attention_layernorm.weight")
        if cfg.is_dense_layer(l):
            x = x + gated(h, sd[p + "mlp.w13_weight"], sd[p + "mlp.w2_weight"])
            continue
        w, best = torch.topk(torch.softmax(h @ sd[p + "gate.weight"].double().T, -1), cfg.top_k, dim=-1)
        if cfg.norm_topk_prob:
            w = w / w.sum(-1, keepdim=True)
        for e in range(cfg.num_experts):
            r, j = (best == e).nonzero(as_tuple=True)
            if len(r):
                x[r] += w[r, j, None] * gated(h[r], sd[p + "experts.w13_weight"][e], sd[p + "experts.w2_weight"][e])
        if cfg.num_shared_experts:
            y = gated(h, sd[p + "shared_expert.w13_weight"], sd[p + "shared_expert.w2_weight"])
            if cfg.shared_expert_gate:
                y = y * torch.sigmoid(h @ sd[p + "shared_expert_gate.weight"].double().T)
            x = x + y
    last = torch.tensor(new, device="cuda").cumsum(0) - 1
    return dict(logits=norm(x[last], "norm.weight") @ sd["lm_head.weight"].double().T, caches=[kv])


def convolve(x, taps):
    """Causal, per channel: the last column of taps [C, n] weighs the row itself."""
    n = taps.shape[1]
    full = torch.cat([x.new_zeros(n - 1, x.shape[1]), x])
    return sum(full[j:j + len(x)] * taps[:, j] for j in range(n))


def recurrence(q, k, v, decay, beta=None, bonus=None, write=None):
    """q, k [T, H, D], v [T, H, V], decay [T, H, D or 1] -> read-outs [T, H, V]."""
    S = q.new_zeros(*k.shape[1:], v.shape[-1])
    out = []
    for t in range(len(q)):
        if bonus is not None:
            now = k[t, :, :, None] * v[t, :, None]
            out.append(torch.einsum("hdv,hd->hv", S + bonus[..., None] * now, q[t]))
            S = decay[t, ..., None] * S + now
            continue
        S = decay[t, ..., None] * S
        u = v[t] if beta is None else beta[t, :, None] * (v[t] - torch.einsum("hdv,hd->hv", S, k[t]))
        S = S + k[t, :, :, None] * (u if write is None else u * write[t, :, None])[:, None]
        out.append(torch.einsum("hdv,hd->hv", S, q[t]))
    return torch.stack(out)


def mix_gla(m, h, w, eps):
    split = lambda n: (h @ w(n).T).view(len(h), m.heads, -1)
    z = (h @ w("a1").T) @ w("a2").T + w("a2.b")
    decay = torch.exp(-softplus(-z).view(len(h), m.heads, m.dim) / m.tau)
    o = rms(recurrence(split("q") * m.dim ** -0.5, split("k"), split("v"), decay), eps) * w("norm")
    return (o.flatten(1) * silu(h @ w("g").T)) @ w("o").T


def mix_delta(m, h, w, eps):
    part = lambda n, heads: silu(convolve(h @ w(n).T, w(n + ".conv"))).view(len(h), heads, -1).repeat_interleave(m.heads // heads, 1)
    unit = lambda x: x / torch.sqrt((x * x).sum(-1, keepdim=True) + 1e-6)
    z = ((h @ w("a1").T) @ w("a2").T + w("dt_bias")).view(len(h), m.heads, m.dim)
    decay = torch.exp(-torch.exp(w("A_log"))[:, None] * softplus(z))
    o = recurrence(unit(part("q", m.kv_heads)) * m.dim ** -0.5, unit(part("k", m.kv_heads)), part("v", m.heads), decay,
                   beta=torch.sigmoid(h @ w("b").T))
    o = (rms(o, eps) * w("norm")).flatten(1)
    return (o * torch.sigmoid((h @ w("g1").T) @ w("g2").T)) @ w("o").T


def mix_wkv(m, h, w, eps):
    before = torch.cat([torch.zeros_like(h[:1]), h[:-1]])
    mixed = lambda n: h + (before - h) * w("mu." + n)
    r, k, v = ((mixed(n) @ w(n).T).view(len(h), m.heads, m.dim) for n in "rkv")
    z = torch.tanh(mixed("w") @ w("w1").T) @ w("w2").T + w("w0")
    o = recurrence(r, k, v, torch.exp(-torch.exp(z)).view(len(h), m.heads, m.dim), bonus=w("u"))
    return (rms(o, eps).flatten(1) * w("norm") * silu(mixed("g") @ w("g").T)) @ w("o").T


def mix_lightning(m, h, w, eps):
    q, k, v = (silu(h @ w(n).T).view(len(h), m.heads, -1) for n in "qkv")
    decay = torch.tensor(m.decay, dtype=torch.float64, device=h.device)[None, :, None].expand(len(h), -1, 1)
    o = recurrence(q, k, v, decay).flatten(1)
    return (rms(o, eps) * w("norm") * torch.sigmoid(h @ w("g").T)) @ w("o").T


def mix_memory(m, h, w, eps):
    q, k, v = ((h @ w(n).T).view(len(h), m.heads, -1) for n in "qkv")
    cap = lambda n: m.gate_cap * torch.tanh((h @ w(n).T + w(n + ".b")) / m.gate_cap)
    i, f = cap("i"), -softplus(-cap("f"))
    top, tops = torch.zeros_like(i[0]), []
    for t in range(len(h)):
        top = torch.maximum(f[t] + top, i[t])
        tops.append(top)
    tops = torch.stack(tops)
    keep = torch.exp(f + torch.cat([torch.zeros_like(tops[:1]), tops[:-1]]) - tops)[..., None]
    # the normaliser is one more column of the memory, whose values are ones
    o = recurrence(q * m.dim ** -0.5, k, torch.cat([v, torch.ones_like(v[..., :1])], -1), keep, write=torch.exp(i - tops))
    o = o[..., :-1] / (torch.maximum(o[..., -1].abs(), torch.exp(-tops)) + 1e-6)[..., None]
    return (rms(o, eps).flatten(1) * w("norm") * torch.sigmoid(h @ w("g").T)) @ w("o").T


def mix_unit(m, h, w, eps):
    u = convolve(h @ w("x").T + w("x.b"), w("conv")) + w("conv.b")
    r, i = (torch.sigmoid(torch.einsum("tbi,boi->tbo", u.view(len(h), m.blocks, -1), w(n)) + w(n + ".b")).flatten(1) for n in ("ra", "ri"))
    log_a = -8.0 * r * softplus(w("lam"))
    a, b = torch.exp(log_a), torch.sqrt(1.0 - torch.exp(2.0 * log_a)) * i * u
    S, out = torch.zeros_like(u[0]), []
    for t in range(len(h)):
        S = a[t] * S + b[t]
        out.append(S)
    return (torch.stack(out) * gelu_tanh(h @ w("y").T + w("y.b"))) @ w("o").T


def mix_latent(m, h, w, eps, pos):
    q, d = (h @ w("q").T).view(len(h), m.heads, -1), h @ w("dkv").T
    c = rms(d[:, :m.kv_rank], eps) * w("dkv.norm")
    k = torch.cat([(c @ w("uk").T).view(len(h), m.heads, -1), rotate(d[:, None, m.kv_rank:], pos, m.rot).expand(-1, m.heads, -1)], -1)
    q = torch.cat([q[..., :m.dim], rotate(q[..., m.dim:], pos, m.rot)], -1)
    o = attend(q, k, (c @ w("uv").T).view(len(h), m.heads, -1), m.scale, pos, m.window, sink=w("sink") if m.sink else None)
    if m.gate:
        o = (o.view(len(h), m.heads, -1) * torch.sigmoid(h @ w("g").T)[..., None]).flatten(1)
    return o @ w("o").T


def mix_attention(m, h, w, eps, pos, kept, i, first):
    """``kept``: keys and values by layer and sequence; ``first``: the values that later layers mix in."""
    part = lambda n, heads: (h @ w(n).T).view(len(h), heads, -1)
    q = part("q", m.heads)
    if m.qk_norm:
        q = rms(q, eps) * w("q.norm")
    if m.q_temp:
        q = q * (1.0 + m.q_temp.coef * torch.log((pos + 1).div(m.q_temp.every, rounding_mode="floor").double() + 1.0))[:, None, None]
    if m.kv_from is None:
        k = part("k", m.kv_heads)
        v = k if m.tied_values else part("v", m.kv_heads)
        k = rotate(rms(k, eps) * w("k.norm") if m.qk_norm else k, pos, m.rot)
        if m.value_norm:
            v = rms(v, eps)
        if m.v_mix:
            v = (1.0 - w("vmix")) * v + w("vmix") * first["v"] if "v" in first else first.setdefault("v", v)
        kept[i] = k, v
    k, v = kept[i if m.kv_from is None else m.kv_from]
    o = attend(rotate(q, pos, m.rot), k, v, m.scale, pos, m.window, m.chunk, m.softcap, w("sink") if m.sink else None)
    if m.gate:
        o = (o.view(len(h), m.heads, -1) * torch.sigmoid(h @ w("g").T)[..., None]).flatten(1)
    return o @ w("o").T


PLAIN = {GatedLinearSpec: mix_gla, ChannelDeltaSpec: mix_delta, WkvSpec: mix_wkv, HeadDecaySpec: mix_lightning,
         MatrixMemorySpec: mix_memory, GatedUnitSpec: mix_unit}


def mix(m, h, w, eps, pos, kept, i, first):
    if isinstance(m, SideBySideSpec):
        sub = lambda side: (lambda n: w(side + n))
        left, right = mix(m.left, h, sub("left."), eps, pos, kept, i, first), mix(m.right, h, sub("right."), eps, pos, kept, i, first)
        return 0.5 * (rms(left, eps) * w("left.out") + rms(right, eps) * w("right.out"))
    if isinstance(m, LatentAttentionSpec):
        return mix_latent(m, h, w, eps, pos)
    if isinstance(m, AttentionSpec):
        return mix_attention(m, h, w, eps, pos, kept, i, first)
    return PLAIN[type(m)](m, h, w, eps)


def feed(layer, h, w):
    act = {"silu": silu, "gelu_tanh": gelu_tanh}
    three = lambda x, p, f: f(x @ w(p + "gate").T, x @ w(p + "up").T) @ w(p + "down").T
    if layer.ff:
        return three(h, "", lambda g, u: act[layer.act](g) * u)
    r = layer.routed
    z = h @ w("router").T
    s = torch.sigmoid(z) if r.scoring == "sigmoid" else torch.softmax(z, -1)
    choice = s + w("correction") if r.correction else s
    if r.groups > 1:
        parts = choice.view(len(h), r.groups, -1)
        best = parts.topk(2, -1).values.sum(-1).topk(r.keep, -1).indices
        closed = torch.ones_like(parts[..., 0], dtype=torch.bool).scatter_(1, best, False)
        choice = parts.masked_fill(closed[..., None], -math.inf).flatten(1)
    ids = choice.topk(r.top, -1).indices
    wts = s.gather(1, ids)
    if r.renormalize:
        wts = wts / wts.sum(-1, keepdim=True)
    wts = wts * r.scale
    out = torch.zeros_like(h)
    clamped = lambda g, u: g.clamp(max=r.limit) * torch.sigmoid(1.702 * g.clamp(max=r.limit)) * (u.clamp(-r.limit, r.limit) + 1.0)
    one = clamped if r.act == "clamped" else lambda g, u: act[r.act](g) * u
    for e in range(r.experts):
        row, j = (ids == e).nonzero(as_tuple=True)
        if len(row):
            scale = wts[row, j, None]
            out[row] += three(h[row] * scale, f"e{e}.", one) if r.weigh_input else scale * three(h[row], f"e{e}.", one)
    return out


def layer_list_logits(cfg, sd, ids):
    """Whole sequences, all rows together where rows do not meet; logits of the last row of each."""
    eps, lens = cfg.rms_norm_eps, [len(t) for t in ids]
    pos = [torch.arange(n, device="cuda") for n in lens]

    def norm(x, n):
        wt = sd[n].double()
        if cfg.block == "parallel" or cfg.layer_norm:
            x = x - x.mean(-1, keepdim=True)
            return rms(x, eps) * wt + (sd[n + ".b"].double() if cfg.layer_norm else 0.0)
        return rms(x, eps) * (1.0 + wt)

    def gate(h, n):
        return torch.sigmoid(h @ sd[n].double().T + sd[n + ".b"].double()) if cfg.residual_gate else 1.0
    x = sd["embed"][torch.cat(ids)].double() * cfg.embed_scale
    if cfg.positions:
        x = x + sd["pos"].double()[torch.cat(pos)]
    kept, first = [{} for _ in ids], [{} for _ in ids]
    for i, layer in enumerate(cfg.layers):
        p = f"l{cfg.weight_layer(i)}."
        w = lambda n: sd[p + "mix." + n].double()
        ff = lambda h: feed(layer, h, lambda n: sd[p + "mlp." + n].double())
        h = norm(x, p + "norm1")
        parts = h.split(lens)
        if cfg.input_conv:
            parts = [t + convolve(t, sd[p + "canon1"].double()) for t in parts]
        y = torch.cat([mix(layer.mixer, t, w, eps, at, kv, i, v) for t, at, kv, v in zip(parts, pos, kept, first)])
        if cfg.block == "parallel":
            x = x + y + ff(h)
        elif cfg.block == "sandwich":
            x = x + norm(y, p + "norm1b")
            x = x + norm(ff(norm(x, p + "norm2")), p + "norm2b")
        else:
            x = x + cfg.residual_mult * gate(h, p + "rg1") * y
            h = norm(x, p + "norm2")
            x = x + cfg.residual_mult * gate(h, p + "rg2") * ff(h)
    last = torch.tensor(lens, device="cuda").cumsum(0) - 1
    return norm(x[last], "final.norm") @ sd["embed" if cfg.tied_head else "head"].double().T * cfg.logit_scale
