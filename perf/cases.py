"""What the engine is asked to do in use, as cases that can be timed and checked: steps of `Engine.forward` / `Engine.prefill`.

Serving a model is two kinds of steps: prompts in chunks, and a token (or a chain of drafted ones) per stream behind a cached context.
The cases are both kinds on the model families of the presets at their real widths, cut to few layers so that three engines fit one GPU,
with the weight and cache formats that are served. (EXL3 and GGUF weights come from checkpoints only and have no case.) Sizes:

* "27b": the dense hybrid of the benchmark, one period of its layers (three Gated DeltaNet, one attention);
* "moe80b": the routed hybrid, one Gated DeltaNet and one attention layer, experts and projections in NVFP4, as it fits one GPU;
* "mla": the first two (dense) layers of the latent-attention model;
* "small": a generic hybrid of width 1024, where the launches count.

`run` is one step; its outputs are the logits that were asked for and the recurrent states that it leaves.
"""
from __future__ import annotations

import dataclasses
import math

import torch

from ferrite_b200.config import EngineConfig, ModelConfig, hybrid_27b, mla_671b, moe_80b, scaled
from ferrite_b200.engine.engine import Engine
from ferrite_b200.engine.executor import Segment

GRID = 2.0 ** -15            # tensor scale of the NVFP4 weights drawn here
E2M1 = (0.0, 0.5, 1.0, 1.5, 2.0, 3.0, 4.0, 6.0)
QUANTISED = ("in_proj", "out_proj", "gate_up", "down", "lm_head", "experts_gate_up", "experts_down", "shared_gate_up", "shared_down")


# ---- cases ----------------------------------------------------------------------------------------------------------

def listed():
    """`context`: tokens of the longest stream before the step (streams are of unequal length); `rows`: new tokens per stream."""
    case = lambda name, model, do, streams, context, rows, weights="bf16", kv="bf16": dict(
        name=name, model=model, do=do, streams=streams, context=context, rows=rows, weights=weights, kv=kv)
    return [
        # a small model (a draft model, a model on the side) decoding one stream: launches and latency
        case("small-decode-1", "small", "decode", 1, 700, 1),
        # the benchmark's headline: one stream
        case("27b-decode-1", "27b", "decode", 1, 2048, 1),
        # a few users at once, among them long conversations
        case("27b-decode-4", "27b", "decode", 4, 8000, 1),
        # a loaded server
        case("27b-decode-24", "27b", "decode", 24, 1500, 1),
        # speculative decoding: sixteen drafted tokens behind the last one, nine of the rows accepted
        case("27b-verify-17", "27b", "verify", 1, 2048, 17),
        # a new prompt of the benchmark's length
        case("27b-prompt-2048", "27b", "prompt", 1, 0, 2048),
        # the next turn of a long conversation, e4m3 cache
        case("27b-turn-1111", "27b", "turn", 1, 12000, 1111, kv="fp8"),
        # 4-bit weights: one stream, and two (the rows that this format's products take at the activations' full precision: with more
        # rows they round the activations to 4 bits themselves, and differently rounded ones cannot be held against each other)
        case("27b-nvfp4-decode-1", "27b", "decode", 1, 2048, 1, weights="nvfp4"),
        case("27b-nvfp4-decode-2", "27b", "decode", 2, 3000, 1, weights="nvfp4"),
        # the routed model: decoding, and a prompt
        case("moe80b-decode-2", "moe80b", "decode", 2, 2000, 1, weights="nvfp4"),
        case("moe80b-prompt-1500", "moe80b", "prompt", 1, 0, 1500, weights="nvfp4"),
        # latent attention: decoding several streams
        case("mla-decode-6", "mla", "decode", 6, 4000, 1),
    ]


def draw(rng):
    log = lambda lo, hi: int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    model, weights = rng.choice([("small", "bf16"), ("27b", "bf16"), ("27b", "bf16"), ("27b", "nvfp4"), ("moe80b", "nvfp4"), ("mla", "bf16")])
    dos = {"small": ["decode", "decode", "prompt"], "moe80b": ["decode", "prompt"], "mla": ["decode"]}.get(
        model, ["decode", "decode", "verify", "prompt", "turn"] if weights == "bf16" else ["decode"])
    do = rng.choice(dos)
    kv = rng.choice(["bf16", "bf16", "fp8"]) if model == "27b" and weights == "bf16" else "bf16"
    streams, context, rows = 1, 0, 1
    if do == "decode":
        streams = log(1, 2 if weights == "nvfp4" else 32 if model == "27b" else 8)
        context = log(64, min(16000, 32000 // streams))
    elif do == "verify":
        rows, context = log(2, 32), log(64, 12000)
    elif do == "prompt":
        rows = log(33, 2048)
    else:
        rows, context = log(33, 2048), log(500, 12000)
    return dict(model=model, do=do, streams=streams, context=context, rows=rows, weights=weights, kv=kv)


def model_of(case) -> ModelConfig:
    if case["model"] == "27b":
        return scaled(hybrid_27b(), 4)
    if case["model"] == "moe80b":
        return dataclasses.replace(scaled(moe_80b(), 2), full_attn_every=2)
    if case["model"] == "mla":
        return scaled(mla_671b(), 2)
    return ModelConfig(name="small", hidden=1024, inter=3072, n_layers=4, head_dim=128, n_q=8, n_kv=2, rotary_dim=32, rope_theta=1e6, lin_k_heads=8,
                       lin_v_heads=8, lin_dk=128, lin_dv=128, vocab=32768, tie_embeddings=False)


def contexts(case):
    """Tokens in every stream's cache before the step."""
    return [max(1, int(case["context"] * (1 - 0.7 * ((i * 0.618) % 1)))) if case["context"] else 0 for i in range(case["streams"])]


def kept(case):
    """Rows of a stream that stay: all, or those of a verify step that are accepted."""
    return (case["rows"] + 1) // 2 if case["do"] == "verify" else case["rows"]


def tokens(case, cfg, seed):
    g = torch.Generator().manual_seed(seed * 7919 + 5)
    return [torch.randint(0, cfg.vocab, (n + case["rows"],), generator=g) for n in contexts(case)]


# ---- weights --------------------------------------------------------------------------------------------------------

def on_grid(t):
    """`t` with every value moved to what NVFP4 can hold: the codes and scales of a 4-bit checkpoint, written out. Blocks hold their
    largest code and the tensor its largest scale, as a quantiser leaves them, so quantising the values gives them back."""
    flat = t.view(-1, t.shape[-1])
    grid = torch.tensor(E2M1, device=t.device)
    mids = (grid[1:] + grid[:-1]) / 2
    step = max(1, (1 << 26) // flat.shape[1])
    for r in range(0, flat.shape[0], step):
        blk = flat[r:r + step].float().view(-1, 16)
        top = blk.abs().amax(1, keepdim=True).clamp_min(1e-9)
        scale = (top / (6 * GRID)).clamp(2.0, 448.0).to(torch.float8_e4m3fn).float()
        if r == 0:
            scale[0] = 448.0
        mag = grid[torch.bucketize(blk.abs() / (scale * GRID), mids)]
        mag.scatter_(1, blk.abs().argmax(1, keepdim=True), 6.0)
        flat[r:r + step] = (mag * scale * GRID * torch.sign(blk)).view(-1, flat.shape[1]).to(t.dtype)
    return t


def make_weights(case, cfg, seed):
    """Seeded bf16 weights of the architecture under the engine's names, with decays from slow to fast and a decided router."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    w = {}

    def normal(name, *shape, std=0.02, dtype=torch.bfloat16):
        w[name] = torch.empty(shape, dtype=dtype, device="cuda").normal_(0, std, generator=g)
        if case["weights"] == "nvfp4" and name.split(".")[-1] in QUANTISED:
            w[name] = on_grid(w[name])

    h = cfg.hidden
    normal("embed", cfg.vocab, h)
    normal("lm_head", cfg.vocab, h)
    normal("final_norm", h)
    for i, kind in enumerate(cfg.layer_kinds):
        p = f"l{i}."
        normal(p + "input_norm", h)
        normal(p + "post_norm", h)
        if kind == "gdn":
            normal(p + "in_proj", cfg.gdn_in_dim, h)
            normal(p + "conv_w", cfg.conv_dim, cfg.conv_k, std=0.4)
            w[p + "A_log"] = torch.empty(cfg.lin_v_heads, device="cuda").uniform_(math.log(0.01), math.log(4.0), generator=g)
            normal(p + "dt_bias", cfg.lin_v_heads, std=0.5, dtype=torch.float32)
            normal(p + "gnorm_w", cfg.lin_dv)
            w[p + "gnorm_w"] += 1
            normal(p + "out_proj", h, cfg.lin_v_heads * cfg.lin_dv)
        elif kind == "attn":
            normal(p + "in_proj", cfg.attn_in_dim, h)
            normal(p + "q_norm", cfg.head_dim)
            normal(p + "k_norm", cfg.head_dim)
            normal(p + "out_proj", h, cfg.n_q * cfg.head_dim)
        else:
            normal(p + "q_a", cfg.q_lora, h)
            normal(p + "q_a_norm", cfg.q_lora)
            normal(p + "q_b", cfg.n_q * (cfg.nope_head_dim + cfg.rope_head_dim), cfg.q_lora)
            normal(p + "kv_a", cfg.kv_lora + cfg.rope_head_dim, h)
            normal(p + "kv_a_norm", cfg.kv_lora)
            normal(p + "kv_b", cfg.n_q * (cfg.nope_head_dim + cfg.v_head_dim), cfg.kv_lora)
            normal(p + "out_proj", h, cfg.n_q * cfg.v_head_dim)
        if cfg.is_moe(i):
            normal(p + "router", cfg.n_experts, h, std=0.1)
            normal(p + "experts_gate_up", cfg.n_experts, 2 * cfg.expert_inter, h)
            normal(p + "experts_down", cfg.n_experts, h, cfg.expert_inter)
            normal(p + "shared_gate_up", 2 * cfg.expert_inter, h)
            normal(p + "shared_down", h, cfg.expert_inter)
            normal(p + "shared_gate", 1, h)
        else:
            normal(p + "gate_up", 2 * ff_width(cfg), h)
            normal(p + "down", h, ff_width(cfg))
    return w


def ff_width(cfg):
    return cfg.dense_inter if cfg.n_experts and cfg.dense_inter else cfg.inter


# ---- a pass ---------------------------------------------------------------------------------------------------------

def prepare(case, seed):
    """An engine with its streams' contexts in the cache, and the tokens of the step."""
    cfg, ctx, toks = model_of(case), contexts(case), None
    longest = max(ctx) + case["rows"]
    ecfg = EngineConfig(n_slots=case["streams"], max_ctx=-(-longest // 1024) * 1024, weight_dtype=case["weights"], kv_dtype=case["kv"])
    eng = Engine(cfg, make_weights(case, cfg, seed), ecfg, device="cuda", seed=seed)
    toks = [t.tolist() for t in tokens(case, cfg, seed)]
    for i, n in enumerate(ctx):
        if n:
            eng.prefill(i, toks[i][:n], greedy=False)
    return {"case": case, "eng": eng, "ctx": ctx, "new": [t[n:] for t, n in zip(toks, ctx)], "keep": [kept(case)] * len(ctx)}


def run(state):
    """A step. Decoding, verifying and turns repeat at the same positions: the recurrent states go on from where the last pass left them."""
    do, eng, ctx, new = state["case"]["do"], state["eng"], state["ctx"], state["new"]
    if do == "prompt":
        eng.reset_slot(0)
        logits = eng.prefill(0, new[0], greedy=False)[0]
    elif do == "verify":
        logits = eng.forward([Segment(i, ctx[i], t, "all") for i, t in enumerate(new)], commit=False, greedy=False)[0]
        eng.commit_verified(state["keep"])
    else:
        logits = eng.forward([Segment(i, ctx[i], t) for i, t in enumerate(new)], greedy=False)[0]
    return {"logits": logits, "rec": list(eng.ex.rec_state.values()), "conv": list(eng.ex.conv_state.values())}


def work(case):
    """Every weight that a row meets is read once (of the experts those that some row picks), the context's cache rows and the recurrent
    states too; products and attention of the new rows."""
    cfg, ctx, n = model_of(case), contexts(case), case["rows"]
    T = n * case["streams"]
    per = 0.5 + 1 / 16 if case["weights"] == "nvfp4" else 2.0
    el = {"bf16": 2.0, "fp8": 1.0}[case["kv"]]
    h, nbytes, flops = cfg.hidden, T * cfg.hidden * 2.0, 0.0
    for i, kind in enumerate(cfg.layer_kinds):
        if kind == "gdn":
            mats = cfg.gdn_in_dim * h + cfg.lin_v_heads * cfg.lin_dv * h
            state = cfg.lin_v_heads * cfg.lin_dk * cfg.lin_dv
            nbytes += case["streams"] * 4.0 * state * (1 if case["do"] == "prompt" else 2)
            flops += T * 6.0 * state
        elif kind == "attn":
            mats = cfg.attn_in_dim * h + cfg.n_q * cfg.head_dim * h
            nbytes += sum(c + n for c in ctx) * 2.0 * cfg.n_kv * cfg.head_dim * el
            flops += sum(c * n + n * n / 2 for c in ctx) * 4.0 * cfg.n_q * cfg.head_dim
        else:
            L, R, qd = cfg.kv_lora, cfg.rope_head_dim, cfg.nope_head_dim + cfg.rope_head_dim
            mats = h * (cfg.q_lora + L + R) + cfg.n_q * (cfg.q_lora * qd + L * (cfg.nope_head_dim + cfg.v_head_dim) + h * cfg.v_head_dim)
            nbytes += sum(c + n for c in ctx) * (L + R) * el
            flops += sum(c * n + n * n / 2 for c in ctx) * 2.0 * cfg.n_q * (2 * L + R)
        if cfg.is_moe(i):
            one = 3 * h * cfg.expert_inter
            met = cfg.n_experts * (1 - (1 - cfg.top_k / cfg.n_experts) ** T)
            nbytes += (met + 1) * one * per + cfg.n_experts * h * 2.0
            flops += 2.0 * T * ((cfg.top_k + 1) * one + cfg.n_experts * h)
        else:
            mats += 3 * h * ff_width(cfg)
        nbytes += mats * per
        flops += 2.0 * T * mats
    wanted = T if case["do"] in ("decode", "verify") else 1
    return {"bytes": nbytes + cfg.vocab * (h * per + wanted * 4.0), "flops": flops + 2.0 * wanted * cfg.vocab * h}


def tolerance(case):
    # bf16 products and activations through two to four layers: the results are 0.01 to 0.022 (logits) off the 64-bit ones
    return {"rel": 0.03, "max": 0.5}


# ---- the same in 64 bits --------------------------------------------------------------------------------------------

def exact(case, seed):
    cfg, ctx, keep = model_of(case), contexts(case), kept(case)
    w = make_weights(case, cfg, seed)
    toks = [t.cuda() for t in tokens(case, cfg, seed)]
    lens = [len(t) for t in toks]
    f, h, eps = torch.float64, cfg.hidden, cfg.eps
    with torch.no_grad():
        x = w["embed"][torch.cat(toks)].to(f)
        rec, conv = [], []
        for i, kind in enumerate(cfg.layer_kinds):
            lw = {k[len(f"l{i}."):]: v for k, v in w.items() if k.startswith(f"l{i}.")}
            hid = norm(x, lw["input_norm"], eps)
            if kind == "mla":
                parts = [hid[a:b] for a, b in spans(lens)]
                o = torch.cat([latent_attention(cfg, lw, p) for p in parts])
            else:
                rows = torch.split(mul(hid, lw["in_proj"]), lens)
                if kind == "attn":
                    o = torch.cat([attention(cfg, lw, p) for p in rows])
                else:
                    got = [delta_net(cfg, lw, p, n + keep) for p, n in zip(rows, ctx)]
                    o = torch.cat([y for y, _, _ in got])
                    rec.append(torch.stack([s for _, s, _ in got]))
                    conv.append(torch.stack([c for _, _, c in got]))
            del hid
            x = x + mul(o, lw["out_proj"])
            del o
            hid = norm(x, lw["post_norm"], eps)
            x = x + (experts(cfg, lw, hid) if cfg.is_moe(i) else glu(hid, lw["gate_up"], lw["down"]))
        ends = torch.tensor(lens).cumsum(0).tolist()
        want = [r for e in ends for r in range(e - (case["rows"] if case["do"] == "verify" else 1), e)]
        logits = mul(norm(x[want], w["final_norm"], eps), w["lm_head"])
    return {"logits": logits, "rec": rec, "conv": conv}


def spans(lens):
    ends = torch.tensor(lens).cumsum(0).tolist()
    return [(e - n, e) for n, e in zip(lens, ends)]


def mul(x, m, rows=4096):
    m = m.to(torch.float64).t()
    return torch.cat([x[r:r + rows] @ m for r in range(0, x.shape[0], rows)])


def norm(x, weight, eps, centred=True):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps) * (weight.to(x.dtype) + (1 if centred else 0))


def silu(x):
    return x * torch.sigmoid(x)


def glu(x, gate_up, down, rows=4096):
    half = gate_up.shape[0] // 2
    gu, dn = gate_up.to(torch.float64).t(), down.to(torch.float64).t()
    out = []
    for r in range(0, x.shape[0], rows):
        y = x[r:r + rows] @ gu
        out.append((silu(y[:, :half]) * y[:, half:]) @ dn)
    return torch.cat(out)


def experts(cfg, lw, x):
    p = torch.softmax(mul(x, lw["router"]), -1)
    top, ids = p.topk(cfg.top_k, -1)
    top = top / top.sum(-1, keepdim=True) * cfg.route_scale
    out = glu(x, lw["shared_gate_up"], lw["shared_down"]) * torch.sigmoid(mul(x, lw["shared_gate"]))
    for e in ids.unique().tolist():
        row, k = (ids == e).nonzero(as_tuple=True)
        out.index_add_(0, row, glu(x[row], lw["experts_gate_up"][e], lw["experts_down"][e]) * top[row, k][:, None])
    return out


def rotated(x, dims, theta):
    """Pairs (i, i + dims / 2) of the first `dims` columns of x [rows, heads, width], rows at positions 0, 1, .."""
    half = dims // 2
    ang = torch.arange(x.shape[0], dtype=x.dtype, device=x.device)[:, None] * theta ** (-torch.arange(half, dtype=x.dtype, device=x.device) / half)
    c, s = ang.cos()[:, None], ang.sin()[:, None]
    a, b = x[..., :half], x[..., half:dims]
    return torch.cat([a * c - b * s, b * c + a * s, x[..., dims:]], -1)


def causal(q, k, v, scale, rows=512):
    """q, k [n, heads, d], v [n, heads, dv] of one sequence."""
    n, out = q.shape[0], []
    for r in range(0, n, rows):
        m = min(rows, n - r)
        s = torch.einsum("qhd,khd->hqk", q[r:r + m], k[:r + m]) * scale
        ahead = torch.arange(r + m, device=q.device)[None] > torch.arange(r, r + m, device=q.device)[:, None]
        out.append(torch.einsum("hqk,khd->qhd", torch.softmax(s.masked_fill(ahead, -math.inf), -1), v[:r + m]))
    return torch.cat(out)


def attention(cfg, lw, proj):
    n, hd, nq, nkv = proj.shape[0], cfg.head_dim, cfg.n_q, cfg.n_kv
    q, k, v = proj.split([cfg.attn_q_dim, nkv * hd, nkv * hd], 1)
    q, gate = q.view(n, nq, -1).split([hd, hd] if cfg.attn_gate else [hd, 0], -1)
    q = rotated(norm(q, lw["q_norm"], cfg.eps), cfg.rotary_dim, cfg.rope_theta)
    k = rotated(norm(k.reshape(n, nkv, hd), lw["k_norm"], cfg.eps), cfg.rotary_dim, cfg.rope_theta)
    o = torch.cat([causal(qs, k[:, j:j + 1].expand_as(qs), v.view(n, nkv, hd)[:, j:j + 1].expand_as(qs), hd ** -0.5)
                   for j, qs in enumerate(q.split(nq // nkv, 1))], 1)
    return (o * torch.sigmoid(gate) if cfg.attn_gate else o).reshape(n, -1)


def latent_attention(cfg, lw, hid):
    n, nq, dn, dr, dv = hid.shape[0], cfg.n_q, cfg.nope_head_dim, cfg.rope_head_dim, cfg.v_head_dim
    q = mul(norm(mul(hid, lw["q_a"]), lw["q_a_norm"], cfg.eps), lw["q_b"]).view(n, nq, dn + dr)
    lat, kr = mul(hid, lw["kv_a"]).split([cfg.kv_lora, dr], 1)
    kv = mul(norm(lat, lw["kv_a_norm"], cfg.eps), lw["kv_b"]).view(n, nq, dn + dv)
    kr = rotated(kr[:, None], dr, cfg.rope_theta)
    out = []
    for a in range(0, nq, 32):
        qs = q[:, a:a + 32]
        qs = torch.cat([qs[..., :dn], rotated(qs[..., dn:], dr, cfg.rope_theta)], -1)
        ks = torch.cat([kv[:, a:a + 32, :dn], kr.expand(n, qs.shape[1], dr)], -1)
        out.append(causal(qs, ks, kv[:, a:a + 32, dn:], (dn + dr) ** -0.5))
    return torch.cat(out, 1).reshape(n, -1)


def delta_net(cfg, lw, proj, keep, chunk=64):
    """Gated rows of one sequence, its state [heads, dk, dv] behind `keep` rows, and the convolution's inputs before row `keep`."""
    n, nk, nv, dk, dv, taps = proj.shape[0], cfg.lin_k_heads, cfg.lin_v_heads, cfg.lin_dk, cfg.lin_dv, cfg.conv_k
    qkv, z, b, a = proj.split([cfg.conv_dim, nv * dv, nv, nv], 1)
    wide = torch.cat([qkv.new_zeros(taps - 1, cfg.conv_dim), qkv])
    cw = lw["conv_w"].to(proj.dtype)
    y = silu(sum(wide[t:t + n] * cw[:, t] for t in range(taps)))
    q, k, v = y.split([nk * dk, nk * dk, nv * dv], 1)
    unit = lambda t: (t * torch.rsqrt(t.square().sum(-1, keepdim=True) + cfg.eps)).repeat_interleave(nv // nk, 1).transpose(0, 1)
    q, k, v = unit(q.reshape(n, nk, dk)) * dk ** -0.5, unit(k.reshape(n, nk, dk)), v.reshape(n, nv, dv).transpose(0, 1)
    log_g = (-lw["A_log"].to(proj.dtype).exp() * torch.nn.functional.softplus(a + lw["dt_bias"].to(proj.dtype))).t()      # [heads, n]
    beta = torch.sigmoid(b).t()
    S, out, state = proj.new_zeros(nv, dk, dv), [], None
    cuts = sorted({*range(0, n, chunk), keep, n})
    eye = torch.eye(chunk, dtype=proj.dtype, device=proj.device)
    for lo, hi in zip(cuts, cuts[1:]):
        m = hi - lo
        Q, K, V, bt, G = q[:, lo:hi], k[:, lo:hi], v[:, lo:hi], beta[:, lo:hi, None], log_g[:, lo:hi].cumsum(1)
        decay = (G[:, :, None] - G[:, None]).masked_fill(torch.ones(m, m, device=proj.device, dtype=torch.bool).triu(1), -math.inf).exp()
        A = (bt * decay * (K @ K.transpose(1, 2))).tril(-1)
        D = torch.linalg.solve_triangular(eye[:m, :m] + A, bt * (V - G.exp()[..., None] * (K @ S)), upper=False, unitriangular=True)
        out.append(G.exp()[..., None] * (Q @ S) + (decay * (Q @ K.transpose(1, 2))) @ D)
        S = G[:, -1].exp()[:, None, None] * S + (K * (G[:, -1:] - G).exp()[..., None]).transpose(1, 2) @ D
        if hi == keep:
            state = S
    y = norm(torch.cat(out, 1).transpose(0, 1), lw["gnorm_w"], cfg.eps, centred=False) * silu(z.reshape(n, nv, dv))
    return y.reshape(n, -1), state, wide[keep:keep + taps - 1]
