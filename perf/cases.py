"""What the engine is measured on: serving passes over its decoders.

A case is one pass of a serving loop: a group of requests is admitted by the scheduler, their prompts run in
steps of at most ``budget`` tokens (prompt portions beside the tokens of requests that already decode), every
request then decodes ``decode`` more tokens in graph-replayed steps, and all of them are finished.  The tokens a
request "chooses" are given in advance, so that every pass runs the same work whatever the logits' last bits are;
the pass returns the float32 logits of every token that was asked for.  Weights are the engine's seeded random ones.

The decoders are those whose every result follows smoothly from its inputs: Qwen3 (the main one: bfloat16, and the
float32 path), Ruvuvik, Feruzen with dense feed-forwards, and Vametar.  The other designs run on the same attention,
product and recurrence kernels behind routers, where a choice that falls the other way by one rounding is another
feed-forward altogether and no tolerance could say how far two correct results may lie apart.  Models of more than a
gigabyte or two are cut to a few of their layers: every layer costs the same.
"""
import math

import numpy as np
import torch

from tinyinfer_b200 import Engine, SamplingParams, StepEntry
from tinyinfer_b200.config.registry import architecture_of
from tinyinfer_b200.engine.scheduler import Request, Scheduler
from tinyinfer_b200.parts.model import CausalLM
from tinyinfer_b200.weights.random_init import random_tensor

F64 = torch.float64
PAGE = 64
DEVICE = "cuda:0"

# ---- the models ---------------------------------------------------------------------------------
# width, heads, kv heads, feed-forward, tied head
QWEN3 = {"0.6b": (1024, 16, 8, 3072, True), "8b": (4096, 32, 8, 12288, False), "32b": (5120, 64, 8, 25600, False)}
QWEN3_VOCAB, VOCAB = 151936, 32768
# width, heads, kv heads, head size, chunk, latent rank, rotated part, feed-forward
RUVUVIK = {"w1024": (1024, 16, 4, 64, 1024, 256, 32, 2816), "w2048": (2048, 16, 4, 128, 2048, 512, 64, 5632)}
# width, heads, kv heads, head size, recurrent heads with key and value size, feed-forward (Feruzen and Vametar)
MIXED = {"w1024": (1024, 16, 4, 64, 8, 64, 128, 2816), "w2048": (2048, 16, 4, 128, 16, 128, 128, 5632)}


def config_of(case):
    model, size, n = case["model"], case["size"], case["layers"]
    if model == "qwen3":
        w, h, g, ff, tied = QWEN3[size]
        return dict(architectures=["Qwen3ForCausalLM"], num_hidden_layers=n, hidden_size=w, num_attention_heads=h,
                    num_key_value_heads=g, head_dim=128, intermediate_size=ff, vocab_size=QWEN3_VOCAB,
                    rope_theta=1000000.0, rms_norm_eps=1e-6, tie_word_embeddings=tied, max_position_embeddings=40960)
    if model == "ruvuvik":
        w, h, g, d, chunk, rank, dr, ff = RUVUVIK[size]
        mlp = {"kind": "dense", "ff": ff}
        kinds = [
            {"type": "attention", "mlp": mlp,
             "mixer": {"heads": h, "kv_heads": g, "dim": d, "vdim": d, "mask": {"size": chunk},
                       "rot": {"dims": d, "base": 10000.0}, "scale": d ** -0.5, "softcap": 50.0}},
            {"type": "latent_attention", "mlp": mlp,
             "mixer": {"heads": h, "dim": d, "rot_dim": dr, "vdim": d, "kv_rank": rank,
                       "rot": {"dims": dr, "base": 100000.0}, "scale": (d + dr) ** -0.5}},
            {"type": "wkv", "mlp": mlp, "mixer": {"heads": w // 64, "dim": 64, "decay_rank": 64}}]
        return {"architecture": "Ruvuvik", "vocab": VOCAB, "width": w, "norm": {"eps": 1e-5}, "layers": kinds * (n // 3)}
    w, h, g, d, rh, rd, rv, ff = MIXED[size]
    heads = {"heads": h, "kv_heads": g, "dim": d, "vdim": d, "rot": {"dims": d, "base": 500000.0}, "scale": d ** -0.5}
    if model == "feruzen":
        mlp = {"kind": "dense", "ff": ff, "limit": 7.0}
        delta = {"type": "delta", "mlp": mlp, "mixer": {"heads": rh, "kv_heads": rh, "dim": rd, "vdim": rv, "conv": 4}}
        sides = {"type": "parallel", "mlp": mlp, "mixer": {
            "left": heads, "right": {"heads": rh, "dim": rd, "vdim": rv, "gate_cap": 15.0},
            "left_scale": 1.0, "right_scale": 1.0}}
        return {"architecture": "Feruzen", "vocab": VOCAB, "width": w, "norm": {"eps": 1e-6, "groups": 1},
                "canon": {"taps": 4}, "layers": [delta, sides, delta] * (n // 3)}
    mlp = {"kind": "dense", "ff": ff}
    kinds = [{"type": "attention", "mlp": mlp, "mixer": dict(heads, v_mix=True)},
             {"type": "rglru", "mlp": mlp, "mixer": {"width": w, "blocks": 8, "conv": 4}},
             {"type": "gla", "mlp": mlp, "mixer": {"heads": rh, "dim": rd, "vdim": rv, "tau": 16.0, "decay_rank": 16}}]
    return {"architecture": "Vametar", "vocab": VOCAB, "width": w, "norm": {"eps": 1e-6}, "residual_mult": 0.7,
            "embedding": {"bigram": {"buckets": 8191, "mul_prev": 1009, "mul_cur": 13}}, "logit_scale": 1.0,
            "layers": kinds * (n // 3)}


def vocab_of(case):
    return QWEN3_VOCAB if case["model"] == "qwen3" else VOCAB


def specs_of(case):
    """Name -> specification of every tensor of the case's model."""
    config = config_of(case)
    arch = architecture_of(config)
    return CausalLM(arch.build_plan(arch.from_dict(config))).expected_tensors()


# ---- the cases ----------------------------------------------------------------------------------
def _case(name, model, size, layers, requests, prompt, decode, dtype="bfloat16", budget=2048):
    case = {"model": model, "size": size, "layers": layers, "dtype": dtype, "requests": requests, "prompt": prompt,
            "decode": decode, "budget": budget}
    return dict({"name": name}, **case) if name else case


def listed():
    return [
        # one user, a short question: what counts is the latency of a single-token step
        _case("0.6b one short chat", "qwen3", "0.6b", 28, 1, 29, 24),
        # eight users with prompts of up to two thousand tokens: the ordinary load
        _case("0.6b eight chats", "qwen3", "0.6b", 28, 8, 1963, 32),
        # many users in small steps: prompt portions beside many decoding requests
        _case("0.6b busy server", "qwen3", "0.6b", 28, 48, 331, 16, budget=512),
        # a long document in portions, a few words about it
        _case("0.6b long document", "qwen3", "0.6b", 28, 1, 20003, 4),
        # the wider models: prompts and a small batch; a full batch of short chats
        _case("8b eight chats", "qwen3", "8b", 6, 8, 1801, 16),
        _case("32b full batch", "qwen3", "32b", 3, 64, 93, 16),
        # the 32-bit path, as replays and comparisons run it: a prompt beside single tokens
        _case("0.6b float32", "qwen3", "0.6b", 8, 3, 197, 8, dtype="float32"),
        # chunked attention, latent attention and a recurrent mixer: a long prompt; a batch that decodes
        _case("ruvuvik long prompt", "ruvuvik", "w2048", 6, 1, 4003, 4),
        _case("ruvuvik eight chats", "ruvuvik", "w1024", 6, 8, 507, 24),
        # delta rule, attention beside a matrix memory
        _case("feruzen chats", "feruzen", "w1024", 6, 4, 1021, 16),
        # attention, a recurrence per channel, gated linear attention
        _case("vametar prompts", "vametar", "w2048", 6, 3, 2011, 8),
        _case("vametar full batch", "vametar", "w1024", 6, 32, 77, 24),
    ]


def prompt_lengths(case):
    """Ragged: the first request has the case's length, the others 40 to 100 % of it."""
    return [max(1, round(case["prompt"] * (1.0 - 0.6 * ((0.618034 * i) % 1.0)))) for i in range(case["requests"])]


def _span(rng, lo, hi):
    """A whole number between lo and hi, spread over the logarithm."""
    return max(lo, min(hi, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def _seconds(case):
    """A pass on a fast card, roughly: what bounds the drawn sizes."""
    w = work(case)
    rate = 4e12 if case["dtype"] == "float32" else 4e14 if case["model"] == "qwen3" else 5e13
    return w["flops"] / rate + w["bytes"] / 3e12


def draw(rng):
    while True:
        model, size, layers = rng.choice([("qwen3", "0.6b", 28), ("qwen3", "0.6b", 28), ("qwen3", "8b", 6), ("qwen3", "32b", 3),
                                          ("ruvuvik", "w1024", 6), ("ruvuvik", "w2048", 6), ("feruzen", "w1024", 6),
                                          ("vametar", "w1024", 6), ("vametar", "w2048", 6)])
        dtype = "float32" if (model, size) == ("qwen3", "0.6b") and rng.random() < 0.25 else "bfloat16"
        if dtype == "float32":
            case = _case(None, model, size, 8, _span(rng, 1, 6), _span(rng, 5, 300), rng.randint(2, 10), dtype)
        else:
            longest = 20000 if size == "0.6b" else 2000 if model != "ruvuvik" else 4000
            case = _case(None, model, size, layers, _span(rng, 1, 64), _span(rng, 3, longest), rng.randint(3, 32),
                         dtype, rng.choice([512, 2048, 2048]))
        if _seconds(case) <= 0.12:
            return case


# ---- a pass -------------------------------------------------------------------------------------
class State:
    def __init__(self, case, seed):
        self.case = case
        lens, extra = prompt_lengths(case), case["decode"]
        g = torch.Generator().manual_seed(seed)
        vocab = vocab_of(case)
        self.prompts = [torch.randint(0, vocab, (n,), generator=g).tolist() for n in lens]
        # the tokens each request goes on with; the last one is chosen and never run
        self.chosen = [torch.randint(0, vocab, (extra + 1,), generator=g).tolist() for _ in lens]
        pages = sum(-(-(n + extra + 1) // PAGE) for n in lens)
        self.engine = Engine(config=config_of(case), seed=seed, dtype=case["dtype"], device=DEVICE, page_size=PAGE,
                             num_pages=pages, max_requests=len(lens))
        self.rows = len(lens) * (extra + 1)
        self.raw = torch.empty((self.rows, vocab), dtype=torch.float32, device=DEVICE)


def prepare(case, seed):
    """An engine with its weights and its decode steps captured, as a server is before its first request."""
    state = State(case, seed)
    run(state)
    torch.cuda.synchronize()
    return state


def run(state):
    """One pass; returns the logits ``[request, token, vocabulary]``."""
    engine, case = state.engine, state.case
    sched = Scheduler(engine.cache, max_num_seqs=case["requests"], max_batched_tokens=case["budget"],
                      max_position=engine.plan.max_position)
    requests = [Request(req_id=("request", i), prompt=p, params=SamplingParams(max_tokens=case["decode"] + 1))
                for i, p in enumerate(state.prompts)]
    for r in requests:
        sched.add(r)
    at, order = 0, []
    while sched.has_work():
        plan = sched.schedule()
        entries = [StepEntry(s.request.req_id, s.request.span(s.start, s.count), [s.count - 1] if s.samples else [])
                   for s in plan]
        if all(s.count == 1 and s.samples for s in plan):
            logits = engine.decode_step(entries)
        else:
            logits = engine.step(entries)
        state.raw[at:at + logits.shape[0]].copy_(logits)
        at += logits.shape[0]
        picked = []
        for s in plan:
            if s.samples:
                number, k = s.request.number, len(s.request.output)
                order.append(number * (case["decode"] + 1) + k)
                picked.append(state.chosen[number][k])
        sched.step_done(plan, picked)
    places = torch.from_numpy(np.argsort(np.asarray(order))).pin_memory().to(DEVICE, non_blocking=True)
    return state.raw.index_select(0, places).view(case["requests"], case["decode"] + 1, -1)


def work(case):
    """Every prompt token through every matrix; a step's weights, and the keys, values and states that a decode
    step needs, read once a step; the logits written."""
    specs = specs_of(case)
    vocab, c = vocab_of(case), config_of(case)
    width = c.get("width") or c["hidden_size"]
    params = sum(math.prod(s.shape) for n, s in specs.items() if len(s.shape) > 1 and "embed" not in n and "head" not in n
                 and n != "bigram")
    lens, extra = prompt_lengths(case), case["decode"]
    tokens, rows = sum(lens) + len(lens) * extra, len(lens) * (extra + 1)
    steps = -(-sum(lens) // case["budget"]) + extra
    flops = 2.0 * params * tokens + 2.0 * vocab * width * rows
    data = 2.0 * (params + vocab * width) * steps + 4.0 * vocab * rows
    if case["model"] == "qwen3":
        layers = [{"type": "attention", "mixer": {"heads": c["num_attention_heads"], "dim": 128,
                                                  "kv_heads": c["num_key_value_heads"]}}] * case["layers"]
    else:
        layers = c["layers"]
    each = 4 if case["dtype"] == "float32" else 2
    for layer in layers:
        m = layer["mixer"]
        sides = [("attention", m["left"]), ("memory", m["right"])] if layer["type"] == "parallel" else [(layer["type"], m)]
        for kind, m in sides:
            if kind in ("attention", "latent_attention"):
                chunk = m["mask"]["size"] if m.get("mask") else 1 << 30
                seen = sum(_seen(n + extra, chunk) for n in lens)
                late = sum(_seen(n + extra, chunk) - _seen(n, chunk) for n in lens)
                if kind == "attention":
                    flops += 4.0 * m["heads"] * m["dim"] * seen
                    data += 2.0 * each * m["kv_heads"] * m["dim"] * late
                else:
                    flops += 2.0 * m["heads"] * (2 * m["dim"] + m["rot_dim"]) * seen
                    data += each * (m["kv_rank"] + m["rot_dim"]) * late
            elif kind == "rglru":
                flops += 10.0 * m["width"] * tokens
                data += 8.0 * m["width"] * len(lens) * extra
            else:
                state = m["heads"] * m["dim"] * m.get("vdim", m["dim"])
                flops += 6.0 * state * tokens
                data += 8.0 * state * len(lens) * extra
    return {"bytes": data, "flops": flops}


def _seen(n, chunk):
    """Keys that ``n`` tokens from the start of a request see in chunks of ``chunk``."""
    whole, rest = divmod(n, chunk)
    return whole * chunk * (chunk + 1) / 2 + rest * (rest + 1) / 2


def tolerance(case):
    """A pass lies this far from the same in 64 bits: bfloat16 0.005 to 0.006 for most decoders, 0.010 to 0.014
    for the widths of 4,096 and 5,120 and 0.013 to 0.016 for Vametar, float32 2.2e-6; the roundings of another order of
    sums are others, so two correct results lie about 1.4 times that apart.  Stated is about four times as much, at most
    0.03; the largest of some million normal errors is five to six times their mean."""
    if case["dtype"] == "float32":
        return {"rel": 1e-5, "max": 1e-4}
    wide = case["size"] in ("8b", "32b") or case["model"] == "vametar"
    return {"rel": 0.03 if wide else 0.024, "max": 0.24 if wide else 0.18}


# ---- the same in 64 bits ------------------------------------------------------------------------
class Weights:
    """The case's tensors in 64 bits, drawn as they are asked for."""

    def __init__(self, case, seed):
        self.specs, self.seed = specs_of(case), seed

    def __getitem__(self, name):
        return random_tensor(self.seed, name, self.specs[name], device=DEVICE).to(F64)


def unit(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def silu(z):
    return z * torch.sigmoid(z)


def attend(q, k, v, scale, chunk=None, cap=None, factor=None, sink=None):
    """Causal attention of q ``[T, H, d]`` over k, v ``[T, G, d]``: inside chunks, with a factor per head and a cap on
    the score, and one logit without a value per head."""
    t, nh, _ = q.shape
    group = nh // k.shape[1]
    kh, vh = (x.transpose(0, 1).repeat_interleave(group, 0) for x in (k, v))
    pos = torch.arange(t, device=q.device)
    out = []
    block = max(16, (1 << 27) // (nh * t))
    for a in range(0, t, block):
        rows = pos[a:a + block]
        end = int(rows[-1]) + 1
        s = (q[a:a + block].transpose(0, 1) @ kh[:, :end].transpose(1, 2)) * scale
        s = s if factor is None else s * factor[:, None, None]
        s = s if cap is None else cap * torch.tanh(s / cap)
        dark = pos[None, :end] > rows[:, None]
        if chunk is not None:
            dark |= pos[None, :end] // chunk != rows[:, None] // chunk
        s = s.masked_fill(dark, -math.inf)
        if sink is not None:
            s = torch.cat([s, sink[:, None, None].expand(nh, s.shape[1], 1)], 2)
        p = torch.softmax(s, -1)[..., :end]
        out.append((p @ vh[:, :end]).transpose(0, 1))
    return torch.cat(out).reshape(t, -1)


def turned(x, dims, base, pairs, angle32=False):
    """The first ``dims`` elements of every head turned, as neighbouring pairs or as halves."""
    pos = torch.arange(x.shape[0], device=x.device, dtype=F64)
    freq = base ** (-2.0 * torch.arange(dims // 2, device=x.device, dtype=F64) / dims)
    ang = (pos.float()[:, None] * freq.float()[None] if angle32 else pos[:, None] * freq[None]).to(F64)[:, None]
    c, s = torch.cos(ang), torch.sin(ang)
    out = x.clone()
    a = x[..., 0:dims:2] if pairs else x[..., :dims // 2]
    b = x[..., 1:dims:2] if pairs else x[..., dims // 2:dims]
    turned_a, turned_b = a * c - b * s, b * c + a * s
    if pairs:
        out[..., 0:dims:2], out[..., 1:dims:2] = turned_a, turned_b
    else:
        out[..., :dims // 2], out[..., dims // 2:dims] = turned_a, turned_b
    return out


def shifted(x, n):
    """Row t of the result is row t - n of x, zeros before the start."""
    return torch.cat([torch.zeros_like(x[:n]), x[:x.shape[0] - n]]) if n < x.shape[0] else torch.zeros_like(x)


def time_conv(x, taps):
    n = taps.shape[1]
    return sum(shifted(x, n - 1 - j) * taps[:, j] for j in range(n))


def walk(t, state, step):
    """``step(i, state)`` gives token i's row and the next state."""
    rows = []
    for i in range(t):
        row, state = step(i, state)
        rows.append(row)
    return torch.stack(rows)


def qwen3_logits(c, w, seqs, firsts):
    nh, g, eps = c["num_attention_heads"], c["num_key_value_heads"], c["rms_norm_eps"]
    table = w["model.embed_tokens.weight"]
    xs = [table[s] for s in seqs]
    del table
    for i in range(c["num_hidden_layers"]):
        p = f"model.layers.{i}."
        n = {k: w[p + k + ".weight"] for k in (
            "input_layernorm", "post_attention_layernorm", "self_attn.q_proj", "self_attn.k_proj", "self_attn.v_proj",
            "self_attn.o_proj", "self_attn.q_norm", "self_attn.k_norm", "mlp.gate_proj", "mlp.up_proj", "mlp.down_proj")}
        for j, x in enumerate(xs):
            h = unit(x, eps) * n["input_layernorm"]
            q, k, v = ((h @ n[f"self_attn.{a}_proj"].T).view(h.shape[0], -1, 128) for a in "qkv")
            q, k = (turned(unit(a, eps) * n[f"self_attn.{b}_norm"], 128, c["rope_theta"], False, True)
                    for a, b in ((q, "q"), (k, "k")))
            x = x + attend(q, k, v, 128 ** -0.5) @ n["self_attn.o_proj"].T
            h = unit(x, eps) * n["post_attention_layernorm"]
            xs[j] = x + (silu(h @ n["mlp.gate_proj"].T) * (h @ n["mlp.up_proj"].T)) @ n["mlp.down_proj"].T
    head = w["model.embed_tokens.weight" if c["tie_word_embeddings"] else "lm_head.weight"]
    norm = w["model.norm.weight"]
    return [(unit(x[f:], eps) * norm) @ head.T for x, f in zip(xs, firsts)]


def wkv(h, w, p, m, eps):
    nh, d, before = m["heads"], m["dim"], shifted(h, 1)
    mix = {a: h + (before - h) * w[p + "mu." + a] for a in "rkvgw"}
    r, k, v = ((mix[a] @ w[p + a].T).view(-1, nh, d) for a in "rkv")
    decay = torch.exp(-torch.exp(torch.tanh(mix["w"] @ w[p + "w1"].T) @ w[p + "w2"].T + w[p + "w0"])).view(-1, nh, d)
    u = w[p + "u"]

    def step(i, s):
        kv = k[i][:, :, None] * v[i][:, None, :]
        return (r[i][:, None] @ (s + u[:, :, None] * kv))[:, 0], decay[i][:, :, None] * s + kv
    out = unit(walk(h.shape[0], torch.zeros(nh, d, d, dtype=F64, device=h.device), step), eps).reshape(h.shape[0], -1)
    return (out * w[p + "norm"] * silu(mix["g"] @ w[p + "g"].T)) @ w[p + "o"].T


def ruvuvik_mixer(h, w, p, layer, eps):
    m, t = layer["mixer"], h.shape[0]
    if layer["type"] == "wkv":
        return wkv(h, w, p, m, eps)
    nh, d = m["heads"], m["dim"]
    if layer["type"] == "attention":
        q, k = (turned((unit(h @ w[p + a].T, eps) * w[p + a + ".norm"]).view(t, -1, d), m["rot"]["dims"], m["rot"]["base"], True)
                for a in "qk")
        out = attend(q, k, (h @ w[p + "v"].T).view(t, -1, m["vdim"]), m["scale"], m["mask"]["size"], m["softcap"], w[p + "temp"])
        out = out.view(t, nh, -1) * torch.sigmoid(h @ w[p + "g"].T)[:, :, None]
    else:
        dr, rank = m["rot_dim"], m["kv_rank"]
        q = (h @ w[p + "q"].T).view(t, nh, d + dr)
        down = h @ w[p + "dkv"].T
        lat = unit(down[:, :rank], eps) * w[p + "dkv.norm"]
        q_rot, k_rot = (turned(a, dr, m["rot"]["base"], True) for a in (q[:, :, d:], down[:, None, rank:]))
        k = torch.cat([(lat @ w[p + "uk"].T).view(t, nh, d), k_rot.expand(-1, nh, -1)], 2)
        out = attend(torch.cat([q[:, :, :d], q_rot], 2), k, (lat @ w[p + "uv"].T).view(t, nh, -1), m["scale"], sink=w[p + "sink"])
    return out.reshape(t, -1) @ w[p + "o"].T


def ruvuvik_logits(c, w, seqs, firsts):
    eps, out = c["norm"]["eps"], []

    def norm(x, name):
        return unit(x, eps) * (1.0 + w[name])

    for s, first in zip(seqs, firsts):
        x = norm(w["embed"][s], "embed.norm")
        for i, layer in enumerate(c["layers"]):
            p = f"l{i}."
            x = x + ruvuvik_mixer(norm(x, p + "norm1"), w, p + "mix.", layer, eps)
            z, act = norm(x, p + "norm2") @ w[p + "mlp.up"].T, w[p + "mlp.act"]
            ap, aq, neg = math.log1p(math.exp(float(act[0]))), 0.5 + math.log1p(math.exp(float(act[1]))), z.clamp(max=0.0)
            x = x + torch.where(z > 0, ap * z * z + 0.5 * z, aq * (torch.expm1(neg) - neg) + 0.5 * z) @ w[p + "mlp.down"].T
        out.append(norm(x[first:], "final.norm") @ w["head"].T)
    return out


def delta_rule(h, w, p, m, eps):
    t, nh, d, dv = h.shape[0], m["heads"], m["dim"], m["vdim"]
    q, k, v = (silu(time_conv(h @ w[p + a].T, w[p + a + ".conv"])).view(t, nh, -1) for a in "qkv")
    q, k = (a / torch.sqrt((a * a).sum(-1, keepdim=True) + 1e-6) for a in (q * 1.0, k))
    q = q * d ** -0.5
    beta = torch.sigmoid(h @ w[p + "b"].T)[:, :, None]
    decay = torch.exp(-torch.exp(w[p + "A_log"]) * torch.nn.functional.softplus(h @ w[p + "a"].T + w[p + "dt_bias"]))[:, :, None, None]

    def step(i, s):
        s = decay[i] * s
        s = s + k[i][:, :, None] * (beta[i] * (v[i] - (k[i][:, None] @ s)[:, 0]))[:, None]
        return (q[i][:, None] @ s)[:, 0], s
    out = unit(walk(t, torch.zeros(nh, d, dv, dtype=F64, device=h.device), step), eps) * w[p + "norm"]
    return (out * silu(h @ w[p + "g"].T).view(t, nh, dv)).reshape(t, -1) @ w[p + "o"].T


def matrix_memory(h, w, p, m, eps):
    t, nh, d, cap = h.shape[0], m["heads"], m["dim"], m["gate_cap"]
    q, k, v = ((h @ w[p + a].T).view(t, nh, -1).transpose(0, 1) for a in "qkv")
    log_i, log_f = (cap * torch.tanh((h @ w[p + a].T + w[p + a + ".b"]) / cap) for a in "if")
    total = torch.nn.functional.logsigmoid(log_f).cumsum(0).T                   # [heads, T]
    rows = []
    pos = torch.arange(t, device=h.device)
    for a in range(0, t, 512):                                                  # the recurrence written out
        e = min(t, a + 512)
        weight = total[:, a:e, None] - total[:, None, :e] + log_i.T[:, None, :e]
        weight = weight.masked_fill(pos[None, :e] > pos[a:e, None], -math.inf)
        top = torch.maximum(weight.amax(-1), total[:, a:e])
        s = torch.exp(weight - top[:, :, None]) * (q[:, a:e] * d ** -0.5 @ k[:, :e].transpose(1, 2))
        rows.append((s @ v[:, :e]) / (torch.maximum(s.sum(-1).abs(), torch.exp(-top)) + 1e-6)[:, :, None])
    out = unit(torch.cat(rows, 1).transpose(0, 1), eps).reshape(t, -1)
    return (out * w[p + "norm"] * torch.sigmoid(h @ w[p + "g"].T)) @ w[p + "o"].T


def feruzen_logits(c, w, seqs, firsts):
    eps, table, out = c["norm"]["eps"], w["embed"], []
    for s, first in zip(seqs, firsts):
        x = table[s]
        results = [x]
        for i, layer in enumerate(c["layers"]):
            p, m, t = f"l{i}.", layer["mixer"], x.shape[0]
            h = x + time_conv(x, w[p + "canon1"])
            if layer["type"] == "delta":
                y = delta_rule(h, w, p + "mix.", m, eps)
            else:
                a, left = p + "mix.left.", m["left"]
                q, k = (turned(unit((h @ w[a + n].T).view(t, -1, left["dim"]), eps) * w[a + n + ".norm"], left["rot"]["dims"],
                               left["rot"]["base"], True) for n in "qk")
                y = attend(q, k, (h @ w[a + "v"].T).view(t, -1, left["vdim"]), left["scale"]) @ w[a + "o"].T
                y = m["left_scale"] * y + m["right_scale"] * matrix_memory(h, w, p + "mix.right.", m["right"], eps)
            x = x + unit(y, eps) * w[p + "norm1"]
            limit = layer["mlp"]["limit"]
            gate, up = (x @ w[p + "mlp.gate"].T).clamp(max=limit), (x @ w[p + "mlp.up"].T).clamp(-limit, limit)
            y = (gate * torch.sigmoid(1.702 * gate) * (up + 1.0)) @ w[p + "mlp.down"].T
            results.append(x + unit(y, eps) * w[p + "norm2"])
            x = sum(f * r for f, r in zip(w[p + "dwa"], results))
        out.append((unit(x[first:], eps) * w["final.norm"]) @ table.T)
    return out


def gelu(z):
    return torch.nn.functional.gelu(z, approximate="tanh")


def vametar_mixer(h, w, p, layer, eps, kept):
    m, t = layer["mixer"], h.shape[0]
    if layer["type"] == "attention":
        q, k = (turned((unit(h @ w[p + a].T, eps) * w[p + a + ".norm"]).view(t, -1, m["dim"]), m["rot"]["dims"], m["rot"]["base"],
                       False) for a in "qk")
        v = h @ w[p + "v"].T
        if kept:
            v = (1.0 - w[p + "vmix"]) * v + w[p + "vmix"] * kept[0]
        else:
            kept.append(v)
        return attend(q, k, v.view(t, -1, m["vdim"]), m["scale"]) @ w[p + "o"].T
    if layer["type"] == "rglru":
        u = time_conv(h @ w[p + "x"].T + w[p + "x.b"], w[p + "conv"]) + w[p + "conv.b"]
        r, i = (torch.sigmoid(torch.einsum("tbi,boi->tbo", u.view(t, m["blocks"], -1), w[p + a]) + w[p + a + ".b"]).reshape(t, -1)
                for a in ("ra", "ri"))
        log_a = -8.0 * r * torch.nn.functional.softplus(w[p + "lam"])
        a, take = torch.exp(log_a), torch.sqrt(-torch.expm1(2.0 * log_a)) * i * u

        def step(n, s):
            s = a[n] * s + take[n]
            return s, s
        return (walk(t, torch.zeros_like(u[0]), step) * gelu(h @ w[p + "y"].T + w[p + "y.b"])) @ w[p + "o"].T
    nh, d, dv = m["heads"], m["dim"], m["vdim"]
    q, k, v = ((h @ w[p + a].T).view(t, nh, -1) for a in "qkv")
    alpha = torch.sigmoid((h @ w[p + "a1"].T) @ w[p + "a2"].T + w[p + "a2.b"]).pow(1.0 / m["tau"]).view(t, nh, d, 1)

    def step(n, s):
        s = alpha[n] * s + k[n][:, :, None] * v[n][:, None]
        return (q[n][:, None] @ s)[:, 0] * d ** -0.5, s
    out = unit(walk(t, torch.zeros(nh, d, dv, dtype=F64, device=h.device), step), eps) * w[p + "norm"]
    return (out.reshape(t, -1) * silu(h @ w[p + "g"].T)) @ w[p + "o"].T


def vametar_logits(c, w, seqs, firsts):
    eps, mult, b, out = c["norm"]["eps"], c["residual_mult"], c["embedding"]["bigram"], []
    for s, first in zip(seqs, firsts):
        pair = (shifted(s, 1) * b["mul_prev"] + s * b["mul_cur"]) % b["buckets"]
        pair[0] = b["buckets"]
        x, kept = w["embed"][s] + w["bigram"][pair], []
        for i, layer in enumerate(c["layers"]):
            p = f"l{i}."
            h = unit(x, eps) * w[p + "norm1"]
            y = vametar_mixer(h + (shifted(h, 1) - h) * w[p + "shift"], w, p + "mix.", layer, eps, kept)
            x = x + mult * y * torch.sigmoid(h @ w[p + "rg1"].T + w[p + "rg1.b"])
            h = unit(x, eps) * w[p + "norm2"]
            y = (gelu(h @ w[p + "mlp.gate"].T) * (h @ w[p + "mlp.up"].T)) @ w[p + "mlp.down"].T
            x = x + mult * y * torch.sigmoid(h @ w[p + "rg2"].T + w[p + "rg2.b"])
        out.append((unit(x[first:], eps) * w["final.norm"]) @ w["head"].T * c["logit_scale"])
    return out


LOGITS = {"qwen3": qwen3_logits, "ruvuvik": ruvuvik_logits, "feruzen": feruzen_logits, "vametar": vametar_logits}


def exact(case, seed):
    lens, extra = prompt_lengths(case), case["decode"]
    g = torch.Generator().manual_seed(seed)
    prompts = [torch.randint(0, vocab_of(case), (n,), generator=g) for n in lens]
    chosen = [torch.randint(0, vocab_of(case), (extra + 1,), generator=g) for _ in lens]
    if case["model"] != "qwen3" and sum(lens) > 12000:         # their recurrences are walked token by token here
        return None
    seqs = [torch.cat([p, c[:-1]]).to(DEVICE) for p, c in zip(prompts, chosen)]
    with torch.no_grad():
        logits = LOGITS[case["model"]](config_of(case), Weights(case, seed), seqs, [n - 1 for n in lens])
    return torch.stack(logits)
