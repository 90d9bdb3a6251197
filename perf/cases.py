"""The work that programs have this framework do, as cases of known size, and the same results in 64 bits.

A pass is one call of the engine: a decode step (one new token for every live sequence, logits and picks back on the host) or
a prompt (the cache emptied, one to several prompts of unequal length run as one batch, logits of their last tokens back).
Models are those of `leafcutterllm_b200.synth`, at full width; where a case has fewer layers than the model, the layers it has
are the model's own and the time of a step is theirs many times over. Weights and tokens come from the seed.

The tokens that a decode step is given are the seed's too, and not the picks of the step before: a program that checks drafts
or forces a template does the same, and two correct implementations that round differently then still do the same work."""
import random

import numpy as np
import torch

import leafcutterllm_b200 as lc
from leafcutterllm_b200 import synth

# name -> (description, cache type, rotation by position, most layers)
GGUF = {
    "tiny": (synth.TINY, "f32", "call_relative", 22),
    "llama7b": (synth.LLAMA7B, "f16", "absolute", 32),
    "llama7b-q4km": (synth.LLAMA7B_Q4KM, "f16", "absolute", 32),
    "mixtral": (synth.MIXTRAL, "f16", "absolute", 8),
}
LAYERED = ("varasun", "nepudra")
VOCAB = 32000
GROWTH = 1024  # tokens that a decode case's sequences may grow by before they start again


def listed():
    def case(name, model, layers, phase, seqs, shortest, longest):
        return {"name": name, "model": model, "layers": layers, "phase": phase, "seqs": seqs, "shortest": shortest, "longest": longest}
    return [
        # one user on the small Q4_0 / Q8_0 model that also runs on the CPU: launches and latency
        case("tiny-decode", "tiny", 22, "decode", 1, 32, 32),
        # a handful of short questions arriving at the same model together
        case("tiny-prompts", "tiny", 22, "prompt", 6, 24, 150),
        # the headline: one user, Llama-2-7B shape in Q4_K, 2048 tokens of context
        case("7b-decode", "llama7b", 32, "decode", 1, 2048, 2048),
        # time to the first token of that user
        case("7b-prompt", "llama7b", 32, "prompt", 1, 2048, 2048),
        # continuous batching: 64 users with 128 to 4096 tokens of context each
        case("7b-batch", "llama7b", 4, "decode", 64, 128, 4096),
        # a few users on a file with the usual mix of types (Q4_K and Q6_K)
        case("q4km-few", "llama7b-q4km", 32, "decode", 3, 300, 1100),
        # a prompt of ordinary, odd length to such a file
        case("q4km-prompt", "llama7b-q4km", 8, "prompt", 1, 777, 777),
        # 16 users of a mixture of experts
        case("mixtral-batch", "mixtral", 4, "decode", 16, 1024, 1024),
        # prompts to a mixture of experts
        case("mixtral-prompts", "mixtral", 4, "prompt", 3, 200, 1024),
        # checkpoint-directory designs in bf16: a long prompt and a batch through the gated delta rule and latent attention ...
        case("varasun-prompt", "varasun", 8, "prompt", 1, 2048, 2048),
        case("varasun-batch", "varasun", 8, "decode", 24, 200, 1500),
        # ... and a batch through the delta rule with separate removal and windowed attention
        case("nepudra-batch", "nepudra", 8, "decode", 8, 500, 2500),
    ]


def draw(rng):
    """A model, a direction, a number of sequences and their lengths: lengths and numbers spread over their logarithm."""
    def spread(lo, hi):
        return int(round(lo * (hi / lo) ** rng.random()))
    model = rng.choice(sorted(GGUF) + list(LAYERED))
    phase = rng.choice(("decode", "prompt"))
    if model in GGUF:
        layers = {"tiny": 22, "llama7b": rng.randint(4, 12), "llama7b-q4km": 8, "mixtral": rng.randint(2, 4)}[model]
    else:
        layers = rng.choice((4, 8))
    if phase == "prompt":
        seqs = spread(1, 8)
        longest = spread(16, 2048 if seqs <= 2 else 1024)
    else:
        seqs = spread(1, 64 if model == "llama7b" and layers <= 6 else 24)
        longest = spread(32, 4096 if seqs <= 8 else 1024)
    shortest = max(8, int(longest * rng.uniform(0.1, 1.0)))
    return {"model": model, "layers": layers, "phase": phase, "seqs": seqs, "shortest": shortest, "longest": longest}


def lengths(case):
    """The sequences' lengths: uniform between the case's ends, the same for every seed."""
    rng = random.Random(case["seqs"] * 7919 + case["longest"] * 31 + case["shortest"])
    n = [rng.randint(case["shortest"], case["longest"]) for _ in range(case["seqs"])]
    n[0] = case["longest"]
    return n


def spec_of(case):
    if case["model"] in GGUF:
        return GGUF[case["model"]][0].with_layers(case["layers"])
    if case["model"] == "varasun":
        return synth.layered_spec("varasun", 4096, "dddaddda"[: case["layers"]], 11008, VOCAB, 32)
    return synth.nepudra_spec("nepudra", 4096, "gngwgngs"[: case["layers"]], 11008, VOCAB, 32, 8)


def prompts_of(case, seed):
    rng = np.random.default_rng([seed, 11])
    return [rng.integers(0, VOCAB, n).tolist() for n in lengths(case)]


def fed_of(case, seed):
    """What a decode case's sequences are given, step after step."""
    return np.random.default_rng([seed, 12]).integers(0, VOCAB, (GROWTH, case["seqs"]))


def weight_seed(seed):
    return 1000 + seed % (1 << 31)


def prepare(case, seed):
    n, cap = case["seqs"], case["longest"] + (GROWTH if case["phase"] == "decode" else 0)
    pool = sum(lengths(case)) + n * ((GROWTH if case["phase"] == "decode" else 0) + 32)
    size = dict(max_seqs=n, max_seq_len=cap, kv_pool_tokens=pool, seed=weight_seed(seed))
    if case["model"] in GGUF:
        _, cache, rope, _ = GGUF[case["model"]]
        eng = synth.build_engine(spec_of(case), kv_dtype=cache, rope_mode=rope, **size)
    else:
        eng = synth.build_layered_engine(spec_of(case), **size)
    state = {"engine": eng, "phase": case["phase"], "ids": list(range(n)), "prompts": prompts_of(case, seed), "at": 0}
    if case["phase"] == "decode":
        state["fed"] = fed_of(case, seed).tolist()
        eng.forward_batch(state["ids"], state["prompts"], want_logits=False)
    return state


def run(state):
    eng, ids = state["engine"], state["ids"]
    if state["phase"] == "prompt":
        eng.kv_clear()
        logits, _ = eng.forward_batch(ids, state["prompts"])
    else:
        if state["at"] == GROWTH:  # the conversations are full: the next ones begin
            eng.kv_clear()
            eng.forward_batch(ids, state["prompts"], want_logits=False)
            state["at"] = 0
        logits, _ = eng.forward_batch(ids, [[t] for t in state["fed"][state["at"]]])
        state["at"] += 1
    return logits  # and not the greedy picks: of 32,000 random logits the two largest are often nearer than rounding


def work(case):
    """Every matrix once (of the experts those that tokens reach), the cache's live rows and states once, logits out; two
    operations per weight and token, and the attention's products."""
    spec, n, decode = spec_of(case), lengths(case), case["phase"] == "decode"
    tokens = len(n) if decode else sum(n)
    per_token, once = 0.0, 0.0  # weights that a token meets; bytes of all that are read
    for name, typ, dims, _ in spec.tensors():
        count = 1
        for d in dims:
            count *= d
        elems, size = lc.QUANT_GEOMETRY[typ]
        row = count / elems * size
        if name in ("token_embd.weight", "embed", "bigram"):
            once += row / dims[-1] * tokens
        elif ".expert." in name:
            e, k = spec.n_experts, spec.top_k
            once += row * (1 - (1 - k / e) ** tokens)
            per_token += count * k / e
        elif name in ("output.weight", "head"):
            once += row
        else:
            once += row
            per_token += count
    head = 4096 * VOCAB if case["model"] != "tiny" else 2048 * VOCAB
    flops = 2.0 * (per_token * tokens + head * len(n))
    once += 4.0 * VOCAB * len(n)
    if case["model"] in GGUF:
        width, size = spec.num_kv_heads * spec.head_dim, 4 if GGUF[case["model"]][1] == "f32" else 2
        once += sum((c + 1 if decode else c) * 2 * width * size * spec.num_layers for c in n)
        flops += sum(4.0 * spec.hidden_size * (c if decode else c * c / 2) * spec.num_layers for c in n)
        return {"bytes": once, "flops": flops}
    for layer in spec.config["layers"]:
        m = layer["mixer"]
        if layer["type"] in ("channel_delta", "general_delta"):
            state = m["heads"] * m["dim"] * m.get("vdim", m["dim"])
            once += 4.0 * state * len(n) * (2 if decode else 1)
            flops += 6.0 * state * tokens
        elif layer["type"] == "latent_attention":
            once += sum(2.0 * (m["kv_rank"] + m["rot_dim"]) * (c + 1 if decode else c) for c in n)
            flops += sum(2.0 * m["heads"] * (m["dim"] + m["rot_dim"] + m["vdim"]) * (c if decode else c * c / 2) for c in n)
        else:
            seen = [min(c, m["mask"]["size"]) if "mask" in m else c for c in n]
            once += sum(2.0 * m["kv_heads"] * (m["dim"] + m["vdim"]) * (s + 1 if decode else c) for s, c in zip(seen, n))
            flops += sum(2.0 * m["heads"] * (m["dim"] + m["vdim"]) * (s if decode else s * (c - s / 2)) for s, c in zip(seen, n))
    return {"bytes": once, "flops": flops}


def tolerance(case):
    # About four times the distance from exact(): f32 throughout 2.4e-6; with the cache in f16, and angles that are f32 at
    # positions in the thousands, 1.5e-4 to 6.5e-4; a token between two experts goes to the other one, 1e-3 to 6.8e-3; bf16 7e-3 to 1.8e-2.
    rel = {"tiny": 1e-5, "llama7b": 2.5e-3, "llama7b-q4km": 2.5e-3, "mixtral": 2.7e-2}.get(case["model"], 3e-2)
    return {"rel": rel, "max": min(0.5, 20 * rel)}


# ---- the same results in 64 bits: plain torch ------------------------------------------------------------------------------------
def raw_tensor(typ, seed, name, dims):
    """The blocks of a synthetic tensor, as the generator of the inputs leaves them."""
    count = int(np.prod(dims))
    out = torch.empty(lc.load().lc_tensor_bytes(typ, count), dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    lc._capi.check(lc.load().lc_synth_tensor_dev(typ, seed, name.encode(), synth.SIGMA, count, out.data_ptr()))
    lc._capi.check(lc.load().lc_dev_sync())
    return out


def halves(b):
    return b.contiguous().view(torch.float16).double()


def scales_k(s):
    """The eight (scale, minimum) pairs of a Q4_K block's twelve bytes."""
    s = s.int()
    low, high = s[:, 0:4], s[:, 4:8]
    sc = torch.cat([low & 63, (s[:, 8:12] & 15) | ((low >> 6) << 4)], 1)
    mn = torch.cat([high & 63, (s[:, 8:12] >> 4) | ((high >> 6) << 4)], 1)
    return sc.double(), mn.double()


def values(typ, raw, rows, cols):
    """A tensor's values, [rows, cols] in 64 bits."""
    if typ == lc.TYPE_F32:
        return raw.view(torch.float32).double().reshape(rows, cols)
    if typ == lc.TYPE_BF16:
        return raw.view(torch.bfloat16).double().reshape(rows, cols)
    b = raw.reshape(-1, lc.QUANT_GEOMETRY[typ][1])
    d = halves(b[:, :2])
    if typ == lc.TYPE_Q8_0:
        v = d * b[:, 2:].view(torch.int8)
    elif typ == lc.TYPE_Q4_0:
        v = d * (torch.cat([b[:, 2:] & 15, b[:, 2:] >> 4], 1).double() - 8)
    elif typ == lc.TYPE_Q4_K:
        sc, mn = scales_k(b[:, 4:16])
        q = b[:, 16:].reshape(-1, 4, 1, 32)
        q = torch.cat([q & 15, q >> 4], 2).reshape(-1, 8, 32)
        v = (d * sc)[:, :, None] * q - (halves(b[:, 2:4]) * mn)[:, :, None]
    elif typ == lc.TYPE_Q6_K:
        d = halves(b[:, 208:210])
        ql, qh = b[:, :128].reshape(-1, 2, 64), b[:, 128:192].reshape(-1, 2, 32)
        low = torch.stack([ql[:, :, :32] & 15, ql[:, :, 32:] & 15, ql[:, :, :32] >> 4, ql[:, :, 32:] >> 4], 2)
        high = torch.stack([(qh >> s) & 3 for s in (0, 2, 4, 6)], 2)
        q = (low | (high << 4)).double() - 32
        v = (d * b[:, 192:208].view(torch.int8)).reshape(-1, 2, 4, 2, 1) * q.reshape(-1, 2, 4, 2, 16)
    else:
        raise ValueError("type %d" % typ)
    return v.reshape(rows, cols)


def rms(x, eps, w=None):
    y = x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps)
    return y if w is None else y * w


def pieces(f, x, most=16384):
    """f on a few rows at a time."""
    return torch.cat([f(p) for p in x.split(most)])


def attend(q, k, v, scale, window=None, cap=None):
    """q: [T, H, D], the last T of the S positions of k [S, G, D] and v [S, G, E]."""
    t, h, s, g = q.shape[0], q.shape[1], k.shape[0], k.shape[1]
    keys, vals = k.permute(1, 2, 0), v.transpose(0, 1)
    out, at = [], torch.arange(s, device="cuda")
    for part, pos in zip(q.split(512), torch.arange(s - t, s, device="cuda").split(512)):
        z = (part.reshape(-1, g, h // g, q.shape[2]).permute(1, 2, 0, 3) @ keys[:, None]) * scale
        if cap is not None:
            z = cap * torch.tanh(z / cap)
        far = at[None] > pos[:, None]
        if window is not None:
            far |= pos[:, None] - at[None] >= window
        p = torch.softmax(z.masked_fill(far, float("-inf")), -1)
        out.append((p @ vals[:, None]).permute(2, 0, 1, 3).reshape(len(pos), h, -1))
    return torch.cat(out)


def exact_gguf(case, seed):
    spec = spec_of(case)
    _, cache, rope_mode, _ = GGUF[case["model"]]
    types = {name: (typ, dims, kind) for name, typ, dims, kind in spec.tensors()}

    def weight(name):
        typ, dims, kind = types[name]
        rows = int(np.prod(dims[1:])) if len(dims) > 1 else 1
        if kind == "ones":
            return torch.ones(rows, dims[0], dtype=torch.float64, device="cuda")
        return values(typ, raw_tensor(typ, weight_seed(seed), name, dims), rows, dims[0])

    tokens = prompts_of(case, seed)
    places = [list(range(len(t))) for t in tokens]
    if case["phase"] == "decode":
        for i, t in enumerate(fed_of(case, seed)[0].tolist()):
            places[i].append(len(tokens[i]) if rope_mode == "absolute" else 0)
            tokens[i] = tokens[i] + [t]
    ends = np.cumsum([len(t) for t in tokens])
    spans = list(zip([0] + ends[:-1].tolist(), ends.tolist()))
    last = torch.tensor(ends - 1, device="cuda")
    pos = torch.tensor(sum(places, []), device="cuda", dtype=torch.float64)
    H, hd, nh, nkv = spec.hidden_size, spec.head_dim, spec.num_heads, spec.num_kv_heads
    x = weight("token_embd.weight")[torch.tensor(sum(tokens, []), device="cuda")]
    angle = pos[:, None] * spec.rope_theta ** (-torch.arange(0, hd, 2, device="cuda", dtype=torch.float64) / hd)
    cos, sin = torch.cos(angle)[:, None], torch.sin(angle)[:, None]

    def turn(z, at):
        u, v = z[..., : hd // 2], z[..., hd // 2 :]
        return torch.cat([u * cos[at] - v * sin[at], u * sin[at] + v * cos[at]], -1)

    def stored(z):
        return z.half().double() if cache == "f16" else z

    def silu_pair(y, p):
        gate, up, down = (weight(p + n).T for n in ("ffn_gate.weight", "ffn_up.weight", "ffn_down.weight"))
        return pieces(lambda r: (torch.nn.functional.silu(r @ gate) * (r @ up)) @ down, y)

    for l in range(spec.num_layers):
        p, final = "blk.%d." % l, l == spec.num_layers - 1
        h = rms(x, 1e-5, weight(p + "attn_norm.weight"))
        every = slice(None)
        k = stored(turn((h @ weight(p + "attn_k.weight").T).reshape(-1, nkv, hd), every))
        v = stored((h @ weight(p + "attn_v.weight").T).reshape(-1, nkv, hd))
        at = last if final else every  # nothing reads the other rows of the last layer
        q = turn((h[at] @ weight(p + "attn_q.weight").T).reshape(-1, nh, hd), at)
        o = torch.cat([attend(q[i : i + 1] if final else q[a:b], k[a:b], v[a:b], hd ** -0.5) for i, (a, b) in enumerate(spans)])
        x = x[at] + o.reshape(-1, nh * hd) @ weight(p + "attn_output.weight").T
        h = rms(x, 1e-5, weight(p + "ffn_norm.weight"))
        if spec.n_experts:
            score, chosen = torch.topk(h @ weight(p + "ffn_gate_inp.weight").T, spec.top_k)
            share = torch.softmax(score, -1)
            for e in range(spec.n_experts):
                row, slot = (chosen == e).nonzero(as_tuple=True)
                if len(row):
                    x = x.index_add(0, row, silu_pair(h[row], "%sexpert.%d." % (p, e)) * share[row, slot, None])
        else:
            x = x + silu_pair(h, p)
    return rms(x, 1e-5, weight("output_norm.weight")) @ weight("output.weight").T


def frequencies(rot):
    """Angle per position of each pair, and the factor on sine and cosine, with the usual blend for stretched contexts."""
    dims, sc = rot["dims"], rot["scaling"]
    i = np.arange(dims // 2)
    f = rot["base"] ** (-2.0 * i / dims)

    def dim_of(turns):
        return dims * np.log(sc["original"] / (2 * np.pi * turns)) / (2 * np.log(rot["base"]))
    lo, hi = max(np.floor(dim_of(sc["fast"])), 0), min(np.ceil(dim_of(sc["slow"])), dims - 1)
    ramp = np.clip((i - lo) / max(hi - lo, 0.001), 0, 1)
    return torch.tensor(f / sc["factor"] * ramp + f * (1 - ramp), device="cuda"), 0.1 * np.log(sc["factor"]) + 1


def rotate(x, rot, halves_apart):
    """x: [B, T, heads, n] from position 0 on; pairs are neighbours, or half a rotation apart."""
    f, size = frequencies(rot)
    a = torch.arange(x.shape[1], device="cuda", dtype=torch.float64)[:, None, None] * f
    cos, sin, n = torch.cos(a) * size, torch.sin(a) * size, rot["dims"]
    u, v = (x[..., : n // 2], x[..., n // 2 : n]) if halves_apart else (x[..., :n:2], x[..., 1:n:2])
    pair = [u * cos - v * sin, v * cos + u * sin]
    return torch.cat([torch.cat(pair, -1) if halves_apart else torch.stack(pair, -1).flatten(-2), x[..., n:]], -1)


def unit(x):
    return x * torch.rsqrt(x.square().sum(-1, keepdim=True) + 1e-6)


def exact_layered(case, seed):
    spec = spec_of(case)
    c, eps = spec.config, spec.config["norm"]["eps"]
    types = {name: (typ, dims, kind) for name, typ, dims, kind in spec.tensors()}

    def weight(name):
        typ, dims, kind = types[name]
        if kind != "normal":
            return torch.full((dims[0],), float(kind == "ones"), dtype=torch.float64, device="cuda")
        w = values(typ, raw_tensor(typ, weight_seed(seed), name, dims), int(np.prod(dims[1:])), dims[0])
        return w if len(dims) > 1 else w[0]

    def linear(x, name):
        w = weight(name).T
        return pieces(lambda r: r @ w, x.reshape(-1, x.shape[-1])).reshape(x.shape[:-1] + (-1,))

    tokens = prompts_of(case, seed)
    if case["phase"] == "decode":
        tokens = [t + [int(n)] for t, n in zip(tokens, fed_of(case, seed)[0])]
    # sequences side by side, the shorter ones filled up behind their ends, where nothing looks
    longest = max(len(t) for t in tokens)
    ids = torch.tensor([t + [0] * (longest - len(t)) for t in tokens], device="cuda")
    last = torch.tensor([len(t) - 1 for t in tokens], device="cuda")
    B, T = ids.shape

    def seen_by(q, k, v, m):
        window = m["mask"]["size"] if "mask" in m else None
        return torch.stack([attend(q[b], k[b], v[b], m["scale"], window, m.get("softcap")) for b in range(B)])

    def channel_delta(p, m, x):
        H, D, E = m["heads"], m["dim"], m["vdim"]

        def shifted(n):
            y, w = linear(x, p + n), weight(p + n + ".conv")
            y = torch.nn.functional.pad(y, (0, 0, m["conv"] - 1, 0))
            return torch.nn.functional.silu(sum(y[:, j : j + T] * w[:, j] for j in range(m["conv"])))
        q, k = (unit(shifted(n).reshape(B, T, H, D)) for n in "qk")
        v = shifted("v").reshape(B, T, H, E)
        beta = torch.sigmoid(linear(x, p + "b"))
        a = (linear(linear(x, p + "a1"), p + "a2") + weight(p + "dt_bias")).reshape(B, T, H, D)
        g = torch.exp(-torch.exp(weight(p + "A_log"))[:, None] * torch.nn.functional.softplus(a, threshold=60))
        o, S = torch.empty_like(v), torch.zeros(B, H, D, E, dtype=torch.float64, device="cuda")
        for t in range(T):
            S *= g[:, t, :, :, None]
            u = beta[:, t, :, None] * (v[:, t] - (k[:, t, :, None] @ S)[:, :, 0])
            S += k[:, t, :, :, None] * u[:, :, None]
            o[:, t] = (q[:, t, :, None] @ S)[:, :, 0] * D ** -0.5
        gate = torch.sigmoid(linear(linear(x, p + "g1"), p + "g2")).reshape(B, T, H, E)
        return linear((rms(o, eps, weight(p + "norm")) * gate).flatten(2), p + "o")

    def latent(p, m, x):
        H, D, R, C = m["heads"], m["dim"], m["rot_dim"], m["kv_rank"]
        q = linear(rms(linear(x, p + "dq"), eps, weight(p + "dq.norm")), p + "uq").reshape(B, T, H, D + R)
        q = torch.cat([q[..., :D], rotate(q[..., D:], m["rot"], False)], -1)
        z = linear(x, p + "dkv")
        lat = rms(z[..., :C], eps, weight(p + "dkv.norm"))
        turned = rotate(z[:, :, None, C:], m["rot"], False).expand(B, T, H, R)
        k = torch.cat([linear(lat, p + "uk").reshape(B, T, H, D), turned], -1)
        return linear(seen_by(q, k, linear(lat, p + "uv").reshape(B, T, H, -1), m).flatten(2), p + "o")

    def general_delta(p, m, x):
        H, D = m["heads"], m["dim"]
        r, k, v = (linear(x, p + n).reshape(B, T, H, D) for n in "rkv")
        w = torch.sigmoid(linear(torch.tanh(linear(x, p + "w1")), p + "w2") + weight(p + "w0"))
        w = torch.exp(-np.exp(-0.5) * w).reshape(B, T, H, D)
        a = torch.sigmoid(linear(x, p + "a") + weight(p + "a.b")).reshape(B, T, H, D)
        e = unit(k)
        o, S = torch.empty_like(v), torch.zeros(B, H, D, D, dtype=torch.float64, device="cuda")
        for t in range(T):
            held = e[:, t, :, None] @ S
            S *= w[:, t, :, :, None]
            S -= (a[:, t] * e[:, t])[..., None] * held
            S += k[:, t, :, :, None] * v[:, t, :, None]
            o[:, t] = (r[:, t, :, None] @ S)[:, :, 0]
        o = rms(o, eps).flatten(2) * weight(p + "norm")
        return linear(o * torch.sigmoid(linear(x, p + "g")), p + "o")

    kept = {}

    def gated_attention(i, kind, p, m, x):
        H, G, D, second = m["heads"], m["kv_heads"], m["dim"], kind == "attention_2"

        def placed(n, heads):
            z = (linear(x, p + n) + weight(p + n + ".b")).reshape(B, T, heads, D)
            if second:
                z = rms(z, eps, weight(p + n + ".norm"))
            return rotate(z, m["rot"], True) if "rot" in m else z
        q = placed("q", H)
        if "q_temp" in m:
            at = torch.arange(T, device="cuda", dtype=torch.float64)
            q = q * (1 + m["q_temp"]["coef"] * torch.log(torch.floor((at + 1) / m["q_temp"]["every"]) + 1))[:, None, None]
        if "kv_from" not in m:
            kept[i] = placed("k", G), (linear(x, p + "v") + weight(p + "v.b")).reshape(B, T, G, -1)
        k, v = kept[m.get("kv_from", i)]
        y = linear((seen_by(q, k, v, m) * torch.sigmoid(linear(x, p + "g"))[..., None]).flatten(2), p + "o")
        return y if second else y + weight(p + "o.b")

    if c["architecture"] == "Varasun":
        x = weight("embed")[ids]
        for i, layer in enumerate(c["layers"]):
            mix = channel_delta if layer["type"] == "channel_delta" else latent
            x = x + rms(mix("l%d.mix." % i, layer["mixer"], x), eps, weight("l%d.norm1" % i))
            y = linear(torch.relu(linear(x, "l%d.mlp.up" % i)).square(), "l%d.mlp.down" % i)
            x = x + rms(y, eps, weight("l%d.norm2" % i))
        x = x[torch.arange(B, device="cuda"), last]
        cap = c["logit_softcap"]
        return cap * torch.tanh(linear(rms(x, eps, weight("final.norm")), "head") * c["logit_scale"] / cap)
    pair = c["embedding"]["bigram"]
    before = torch.cat([torch.zeros_like(ids[:, :1]), ids[:, :-1]], 1)
    row = (before * pair["mul_prev"] + ids * pair["mul_cur"]) % pair["buckets"]
    row[:, 0] = pair["buckets"]
    x = weight("embed")[ids] + weight("bigram")[row]
    depth = [x]
    for i, layer in enumerate(c["layers"]):
        p = "l%d." % i
        h = rms(x, eps) * weight(p + "norm1")
        x = x + (general_delta(p + "mix.", layer["mixer"], h) if layer["type"] == "general_delta"
                 else gated_attention(i, layer["type"], p + "mix.", layer["mixer"], h))
        h = rms(x, eps) * weight(p + "norm2")
        x = x + linear(torch.nn.functional.gelu(linear(h, p + "mlp.gate"), approximate="tanh") * linear(h, p + "mlp.up"), p + "mlp.down")
        depth.append(x)
        x = sum(w * y for w, y in zip(weight(p + "dwa"), depth))
    x = x[torch.arange(B, device="cuda"), last]
    return linear(rms(x, eps) * weight("final.norm"), "head")


def exact(case, seed):
    return exact_gguf(case, seed) if case["model"] in GGUF else exact_layered(case, seed)
