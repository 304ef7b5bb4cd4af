"""Performance cases of the token-generation framework: requests as a serving program makes them.

A pass is one request on a cache table that the program keeps: the table is emptied, the prompts are ingested and some
tokens are generated. The models are the workloads of `synthetic.CONFIGS` (the two largest with fewer layers, so that a
pass stays below a second; widths, heads and vocabulary are theirs) and the two designs of listed layers at the sizes
that `bench_layered.py` measures. They are loaded once per process, as a serving program does.

Weights are random but conditioned like trained ones: the query norm carries the attention's scale, the norms behind the
sublayers are small, and the output matrix points back at the embeddings, so that the next token has a clear margin (the
same token for a tied matrix, a fixed permutation of the vocabulary for a separate one). Correct implementations then pick
the same tokens.
"""
import importlib
import math
import zlib

import numpy as np
import torch

pkg = importlib.import_module("oxide-beta_b200")
syn = pkg.synthetic

DEVICE = "cuda:0"


# ---- models -----------------------------------------------------------------------------------------------------------

def model_config(model: str, layers: int) -> dict:
    """c1 .. c5: Gemma 4 workloads; pabovik / nozurax: listed layers, width 2560 and 4096."""
    if model in syn.CONFIGS:
        return syn.scaled_down(syn.workload(model)["cfg"], layers=layers)
    width, heads, ff, q_rank = (2560, 16, 10240, 1024) if model == "pabovik" else (4096, 32, 14336, 1536)
    decay = [float(np.exp(-2.0 ** (-8.0 * (h + 1) / (width // 128)))) for h in range(width // 128)]
    mlp = {"kind": "dense", "ff": ff}
    if model == "pabovik":
        kinds = [{"type": "wkv", "mixer": {"heads": width // 64, "dim": 64}, "mlp": mlp},
                 {"type": "latent_attention", "mlp": mlp,
                  "mixer": {"heads": heads, "dim": 128, "vdim": 128, "q_rank": q_rank, "kv_rank": 512, "rot_dim": 64,
                            "rot": {"dims": 64, "base": 10000.0}, "scale": 192 ** -0.5}},
                 {"type": "lightning", "mlp": mlp, "mixer": {"heads": width // 128, "dim": 128, "vdim": 128, "decay": decay}}]
    else:
        kinds = [{"type": "attention", "mlp": mlp,
                  "mixer": {"heads": width // 128, "kv_heads": width // 512, "dim": 128, "vdim": 128, "scale": 128 ** -0.5,
                            "q_temp": {"coef": 0.1, "every": 8192}}},
                 {"type": "retention", "mlp": mlp,
                  "mixer": {"heads": width // 128, "dim": 128, "vdim": 128, "decay": decay, "rot": {"dims": 128, "base": 10000.0}}}]
    return {"architecture": "Pabovik" if model == "pabovik" else "Nozurax", "vocab": 65536, "width": width,
            "norm": {"eps": 1e-6}, "layers": [kinds[i % len(kinds)] for i in range(layers)]}


def is_gemma(model: str) -> bool:
    return model in syn.CONFIGS


def vocab_of(model: str, cfg: dict) -> int:
    return cfg["vocab_size"] if is_gemma(model) else cfg["vocab"]


def weight_list(model: str, cfg: dict):
    return syn.weight_names(cfg) if is_gemma(model) else syn.layered_weight_names(cfg, low_rank=64)


def successor(model: str, cfg: dict, token):
    """The token that the model's output matrix points at from `token`."""
    return token if is_gemma(model) else (np.asarray(token, dtype=np.int64) * 40503 + 1) % vocab_of(model, cfg)


def weight(model: str, name: str, shape, kind: str) -> torch.Tensor:
    """One tensor of a model, the same every time: BF16 on the GPU (f32 for the f32 workload)."""
    if name == "head":                                   # row successor(v) is the embedding of v, scaled
        V, H = shape
        out = torch.empty(shape, dtype=torch.bfloat16, device=DEVICE)
        v = torch.arange(V, device=DEVICE)
        out[(v * 40503 + 1) % V] = (weight(model, "embed", shape, "matrix").float() * H ** -0.5).to(torch.bfloat16)
        return out
    gen = torch.Generator(device=DEVICE).manual_seed(zlib.crc32((model + "/" + name).encode()))
    a = torch.empty(shape, dtype=torch.float32, device=DEVICE)
    if kind == "matrix":
        a.normal_(generator=gen)
        if is_gemma(model):
            a *= 0.02
        elif name != "embed":
            a *= shape[-1] ** -0.5
            if model == "nozurax" and name.endswith((".o", ".down")):
                a *= 0.3                                 # no norm behind the sublayers: small output matrices instead
    elif kind == "mu":
        a.uniform_(0.0, 1.0, generator=gen)
    elif kind == "w0":
        a.uniform_(-6.0, 0.5, generator=gen)
    else:
        a.normal_(generator=gen)
        if kind in ("ones", "norm"):
            a = 1.0 + 0.1 * a
            if "layer_scalar" in name:
                a.fill_(1.0)
            elif "q_norm" in name:
                a *= 2.0 * shape[-1] ** -0.5
            elif name.endswith(("post_attention_layernorm.weight", "post_feedforward_layernorm.weight", "norm1b", "norm2b")):
                a *= 0.25
        else:
            a *= 0.2
    return a if dtype_of(model) == "f32" else a.to(torch.bfloat16)


def dtype_of(model: str) -> str:
    return syn.CONFIGS[model]["dtype"] if is_gemma(model) else "bf16"


_models = {}


def load(model: str, layers: int):
    if (model, layers) not in _models:
        cfg = model_config(model, layers)

        def host():
            for name, shape, kind in weight_list(model, cfg):
                w = weight(model, name, shape, kind)
                yield name, w.cpu().numpy() if w.dtype == torch.float32 else w.view(torch.int16).cpu().numpy().view(np.uint16)
        if is_gemma(model):
            state = pkg.Gemma4CudaState.load(pkg.Gemma4TextConfig(cfg), host(), 0, pkg.F32 if dtype_of(model) == "f32" else pkg.BF16)
        else:
            cls = pkg.models.model_class(cfg)
            state = cls.STATE.load(cls.CONFIG(cfg), host(), 0, pkg.BF16)
        torch.cuda.empty_cache()
        _models[model, layers] = cfg, state
    return _models[model, layers]


# ---- cases ------------------------------------------------------------------------------------------------------------
# call   greedy: prompt -> logits, then the device-resident greedy loop and one step with logits
#        serve:  the same without the prompts' logits: the last prompt tokens start the loop (batches)
#        topk:   prompt -> logits, then one candidate list of 40 per token with a repetition penalty, the host picks
#        turns:  the prompt comes in three portions with an answer of `steps` tokens behind each (logits of every token)
# prompt: tokens of the longest prompt; ragged: the others are shorter, down to an eighth of it

def _case(name, model, layers, batch, prompt, steps, call, kv="bf16", ragged=False):
    c = dict(model=model, layers=layers, batch=batch, prompt=prompt, steps=steps, call=call, kv=kv, ragged=ragged)
    return dict(c, name=name) if name else c


def listed():
    return [
        # the smallest call: the f32 test-size model answers a short prompt; launches and latency are all that counts
        _case("tiny_f32", "c1", 2, 1, 16, 32, "greedy", "f32"),
        # a chat turn on the ~1B model with the default f32 cache, one candidate list per token (the reference's generate loop)
        _case("chat_1b", "c2", 26, 1, 512, 48, "topk", "f32"),
        # a conversation: odd portions into a filled cache, short answers
        _case("turns_1b", "c2", 26, 1, 301, 8, "turns"),
        # the headline: one sequence on the ~4B model, generation weighs most
        _case("decode_4b", "c3", 34, 1, 256, 96, "greedy"),
        # the other direction: a long prompt on the ~4B model for one token
        _case("prompt_4b", "c3", 34, 1, 2048, 1, "greedy"),
        # a few users at once: small batch, unequal prompts
        _case("few_4b", "c3", 34, 4, 333, 48, "serve", ragged=True),
        # a batch on the ~4B model
        _case("batch16_4b", "c3", 34, 16, 500, 64, "serve"),
        # the ~12B widths with 32 sequences, prompts beyond the window
        _case("batch32_12b", "c4", 12, 32, 1100, 64, "serve", ragged=True),
        # the ~27B widths with 64 sequences, unequal prompts: the largest
        _case("batch64_27b", "c5", 6, 64, 777, 32, "serve", ragged=True),
        # listed layers, latent attention / lightning / time mixing: long prompt and an answer
        _case("pabovik_prompt", "pabovik", 12, 1, 3001, 64, "greedy"),
        # the same with a batch of short requests
        _case("pabovik_batch", "pabovik", 12, 32, 150, 64, "serve", ragged=True),
        # listed layers, retention / attention with a sink: one long request
        _case("nozurax_chat", "nozurax", 12, 1, 3000, 64, "greedy"),
    ]


# model, layers, largest batch, longest prompt, most prompt tokens together, most steps, calls, cache types
RANGES = [
    ("c1", 2, 4, 200, 400, 64, ("greedy", "topk", "turns"), ("f32", "bf16")),
    ("c2", 26, 8, 2048, 4096, 64, ("greedy", "topk", "turns", "serve"), ("f32", "bf16")),
    ("c3", 34, 32, 2048, 8192, 96, ("greedy", "turns", "serve"), ("bf16",)),
    ("c4", 12, 64, 2048, 16384, 64, ("serve",), ("bf16",)),
    ("c5", 6, 64, 1024, 24576, 32, ("serve",), ("bf16",)),
    ("pabovik", 12, 64, 4096, 6144, 64, ("greedy", "turns", "serve"), ("bf16",)),
    ("nozurax", 12, 64, 4096, 8192, 64, ("greedy", "turns", "serve"), ("bf16",)),
]


def _spread(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.49)))))))


def _cost(c):
    w = work(c)
    return max(w["bytes"], w["flops"] / 50)


def draw(rng):
    most = max(_cost(c) for c in listed())
    while True:
        model, layers, batch, prompt, tokens, steps, calls, kv = rng.choice(RANGES)
        call = rng.choice(calls)
        B = _spread(rng, 1, batch)
        if call != "serve":
            B = min(B, 4)
        if call in ("topk", "turns"):
            B = 1
        P = _spread(rng, 12, max(12, min(prompt, tokens // B)))
        c = _case(None, model, layers, B, P, _spread(rng, 1, steps if call != "turns" else 12), call, rng.choice(kv), B > 1 and rng.random() < 0.5)
        if _cost(c) <= most:
            return c


def lengths(case):
    B, P = case["batch"], case["prompt"]
    if not case["ragged"]:
        return [P] * B
    return [P] + syn.ragged_lengths(B - 1, max(2, P // 8), P, seed=2).tolist()


def portions(case):
    """Sizes of the three parts of a conversation's prompt."""
    P = case["prompt"]
    a, b = max(1, P // 2), max(1, P // 3)
    return [a, b, max(1, P - a - b)]


def prepare(case, seed):
    cfg, state = load(case["model"], case["layers"])
    lens = lengths(case)
    rounds = 3 if case["call"] == "turns" else 1
    table = state.new_cache_table([n + rounds * (case["steps"] + 1) + 4 for n in lens], batch=case["batch"],
                                  kv_dtype=pkg.F32 if case["kv"] == "f32" else pkg.BF16)
    prompts = _prompts(case, cfg, seed)
    return dict(case=case, cfg=cfg, state=state, table=table, prompts=prompts, lens=lens)


def _prompts(case, cfg, seed):
    rng = np.random.default_rng([seed, case["prompt"], case["batch"]])
    return [rng.integers(0, vocab_of(case["model"], cfg), n).astype(np.uint32) for n in lengths(case)]


def run(s):
    case, state, table, prompts, lens = s["case"], s["state"], s["table"], s["prompts"], s["lens"]
    steps = case["steps"]
    table.reset()
    if case["call"] == "serve":
        if min(lens) > 1:
            state.prefill_prompt(np.concatenate([p[:-1] for p in prompts]), table, lens=[n - 1 for n in lens], want_logits=False)
        ids, _ = state.decode_greedy([p[-1] for p in prompts], table, steps)
        return {"ids": ids, "last": state.decode_token(ids[-1], table)}
    if case["call"] == "turns":
        out, at = [], 0
        for n in portions(case):
            tok = state.extend(prompts[0][at:at + n], table, want=[n - 1])[0]
            out.append(tok)
            for _ in range(steps):
                out.append(state.decode_token(int(out[-1].argmax()), table))
            at += n
        return {"logits": np.stack(out)}
    logits = state.prefill_prompt(np.concatenate(prompts), table, lens=lens)
    first = np.atleast_2d(logits).argmax(-1).astype(np.uint32)
    if case["call"] == "topk":
        # the candidates' ids behind the first are left out: scores that tie to within the rounding may swap places
        tok, ids, scores = int(first[0]), [], []
        for _ in range(steps):
            cand = state.decode_topk(tok, table, 40, 1.1, True)
            tok = cand[0][0]
            ids.append(tok)
            scores.append([score for _, score in cand])
        return {"logits": logits, "ids": np.array(ids), "scores": np.array(scores, dtype=np.float32)}
    ids, _ = state.decode_greedy(first, table, steps)
    return {"logits": logits, "ids": ids, "last": state.decode_token(ids[-1], table)}


# ---- what a pass cannot do without --------------------------------------------------------------------------------------

def _layer_sizes(model, cfg):
    """Per layer: (projection weights, attention: (multiply-adds per token and visible position, K/V values per position,
    window) or None, recurrent state values)."""
    out = []
    if is_gemma(model):
        H, I, D, Nq, Nkv = (cfg[k] for k in ("hidden_size", "intermediate_size", "head_dim", "num_attention_heads", "num_key_value_heads"))
        for t in cfg["layer_types"]:
            window = cfg["sliding_window"] if t == "sliding_attention" else 1 << 30
            out.append((H * (Nq + 2 * Nkv) * D + Nq * D * H + 3 * H * I, (2 * Nq * D, 2 * Nkv * D, window), 0))
        return out
    H = cfg["width"]
    for layer in cfg["layers"]:
        c, t, ff = layer["mixer"], layer["type"], layer["mlp"]["ff"]
        h, d = c["heads"], c["dim"]
        v, w = c.get("vdim", c["dim"]), 3 * H * ff
        if t == "attention":
            kvh = c["kv_heads"]
            out.append((w + H * (h * d + kvh * (d + v) + h * v), (h * (d + v), kvh * (d + v), 1 << 30), 0))
        elif t == "latent_attention":
            r = c["kv_rank"] + c["rot_dim"]
            w += H * (c["q_rank"] + r + 2 * h * v) + c["q_rank"] * h * (d + c["rot_dim"]) + h * (d + v) * c["kv_rank"]
            out.append((w, (h * (r + c["kv_rank"]), r, 1 << 30), 0))
        elif t == "wkv":
            out.append((w + H * (5 * h * d + 64) + 64 * h * d, None, h * d * d))
        else:
            out.append((w + H * (2 * h * d + 3 * h * v), None, h * d * v))
    return out


def work(case):
    model = case["model"]
    cfg = model_config(model, case["layers"])
    V = vocab_of(model, cfg)
    H = cfg["hidden_size"] if is_gemma(model) else cfg["width"]
    es, kvs = 4 if dtype_of(model) == "f32" else 2, 4 if case["kv"] == "f32" else 2
    lens, B, steps = np.array(lengths(case)), case["batch"], case["steps"]
    # passes over the weights: (rows per sequence, start positions, rows whose logits are needed)
    if case["call"] == "turns":
        passes, at = [], 0
        for n in portions(case):
            passes.append((np.array([n]), np.array([at]), 1))
            passes += [(np.array([1]), np.array([at + n + i]), 1) for i in range(steps)]
            at += n + steps
    elif case["call"] == "serve":
        passes = ([(lens - 1, 0 * lens, 0)] if lens.min() > 1 else []) + [(np.ones(B, int), lens - 1 + i, B) for i in range(steps + 1)]
    else:
        passes = [(lens, 0 * lens, B)] + [(np.ones(B, int), lens + i, B) for i in range(steps + (case["call"] == "greedy"))]
    nbytes = flops = 0.0
    sizes = _layer_sizes(model, cfg)
    kinds = {}
    for s in sizes:
        kinds[s] = kinds.get(s, 0) + 1
    for rows, start, heads in passes:
        R = float(rows.sum())
        for (weights, attn, state), count in kinds.items():
            nbytes += count * weights * es
            flops += count * 2.0 * weights * R
            if attn:
                per, values, window = attn
                first = np.minimum(start + 1, window)
                last = np.minimum(start + rows, window)
                seen = float(((first + last) / 2.0 * rows).sum())                     # visible positions, all rows
                read = float(np.minimum(start, window).sum() + R)                     # K/V rows read or written once
                nbytes += count * read * values * kvs
                flops += count * 2.0 * per * seen
            if state:
                nbytes += count * 8.0 * state * B
                flops += count * 6.0 * state * R
        if heads:
            nbytes += V * H * es + 4.0 * heads * V
            flops += 2.0 * V * H * heads
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    # BF16 operands (projection inputs rounded once, f32 sums): two orders of the same sums differ in which way single
    # inputs round, and the layers carry that on
    if dtype_of(case["model"]) == "f32" and case["kv"] == "f32":
        return {"rel": 2e-5, "max": 1e-3, "differ": 0.0}
    return {"rel": 0.02, "max": 0.2, "differ": 0.005}


# ---- the same in 64 bits, plain torch -----------------------------------------------------------------------------------

def _norm(x, w, eps):
    y = x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)
    return y if w is None else y * w


def _rows(f, x, block=8192):
    return torch.cat([f(x[i:i + block]) for i in range(0, x.shape[0], block)])


def _attend(q, k, v, window, scale, sink=None):
    """q [n, heads, D], k, v [n, kv heads, D]: causal attention, a token sees the last `window` positions up to its own."""
    n, heads = q.shape[:2]
    g = heads // k.shape[1]
    out = torch.empty(n, heads, v.shape[2], dtype=q.dtype, device=q.device)
    for i in range(0, n, 512):
        j, lo = min(n, i + 512), max(0, i + 1 - window)
        kk, vv = k[lo:j].repeat_interleave(g, 1), v[lo:j].repeat_interleave(g, 1)
        s = torch.einsum("thd,shd->hts", q[i:j], kk) * scale
        t, p = torch.arange(i, j, device=q.device)[:, None], torch.arange(lo, j, device=q.device)[None]
        s.masked_fill_(((p > t) | (p <= t - window))[None], -math.inf)
        if sink is not None:
            s = torch.cat([s, sink[:, None, None].expand(heads, j - i, 1)], 2)
        a = torch.softmax(s, -1)
        out[i:j] = torch.einsum("hts,shd->thd", a[..., :j - lo], vv)
    return out


def _turn(x, angles, interleaved):
    """x [n, heads, 2 * m], angles [n, m]: pairs (i, i + m), or (2i, 2i + 1), are rotated."""
    c, s = torch.cos(angles)[:, None], torch.sin(angles)[:, None]
    if interleaved:
        u, v = x[..., 0::2], x[..., 1::2]
        return torch.stack([u * c - v * s, v * c + u * s], -1).flatten(-2)
    m = x.shape[-1] // 2
    u, v = x[..., :m], x[..., m:]
    return torch.cat([u * c - v * s, v * c + u * s], -1)


def _angles(n, dims, base):
    f = float(base) ** (-torch.arange(0, dims, 2, dtype=torch.float64, device=DEVICE) / dims)
    return torch.arange(n, dtype=torch.float64, device=DEVICE)[:, None] * f


def _gelu(x):
    return 0.5 * x * (1.0 + torch.tanh(0.7978845608028654 * (x + 0.044715 * x ** 3)))


def _each(seqs, f, *xs):
    """f over every sequence's rows of the stacked xs."""
    return torch.cat([f(*(x[a:b] for x in xs)) for a, b in seqs])


def _decayed(q, k, v, decay, block=64):
    """S_t = decay S_(t-1) + k_t v_t^T, o_t = S_t^T q_t, a block of tokens at a time."""
    n, H, D = q.shape
    S = torch.zeros(H, D, v.shape[2], dtype=q.dtype, device=q.device)
    out = torch.empty(n, H, v.shape[2], dtype=q.dtype, device=q.device)
    for i in range(0, n, block):
        a, b, c = q[i:i + block], k[i:i + block], v[i:i + block]
        m = a.shape[0]
        t = torch.arange(m, dtype=q.dtype, device=q.device)
        gap = t[:, None] - t[None]
        pw = torch.where(gap[None] >= 0, decay[:, None, None] ** gap.clamp(min=0)[None], torch.zeros((), dtype=q.dtype, device=q.device))
        out[i:i + m] = torch.einsum("hts,shv->thv", torch.einsum("thd,shd->hts", a, b) * pw, c) \
            + torch.einsum("thd,hdv->thv", a, S) * (decay[None] ** (t[:, None] + 1))[..., None]
        S = S * (decay ** m)[:, None, None] + torch.einsum("shd,shv->hdv", b * (decay[None] ** (m - 1 - t)[:, None])[..., None], c)
    return out


def _wkv_scan(r, k, v, w, u):
    n, H, D = r.shape
    S = torch.zeros(H, D, D, dtype=r.dtype, device=r.device)
    out = torch.empty_like(v)
    bonus = (r * u[None] * k).sum(-1, keepdim=True) * v
    for t in range(n):
        out[t] = torch.bmm(r[t][:, None], S)[:, 0]
        S = torch.baddbmm(S * w[t][:, :, None], k[t][:, :, None], v[t][:, None])
    return out + bonus


def _mixer(layer, W, h, seqs, eps):
    c, t = layer["mixer"], layer["type"]
    n, H, D = h.shape[0], c["heads"], c["dim"]
    V = c.get("vdim", D)
    if t == "wkv":
        prev = _each(seqs, lambda x: torch.cat([torch.zeros_like(x[:1]), x[:-1]]), h)
        mix = {s: h + (prev - h) * W("mix.mu." + s) for s in "rkvgw"}
        r, k, v = ((mix[s] @ W("mix." + s).T).view(n, H, D) for s in "rkv")
        w = torch.exp(-torch.exp(torch.tanh(mix["w"] @ W("mix.w1").T) @ W("mix.w2").T + W("mix.w0"))).view(n, H, D)
        u = W("mix.u")
        o = _each(seqs, lambda *a: _wkv_scan(*a, u), r, k, v, w)
        g = mix["g"] @ W("mix.g").T
        return (_norm(o, None, eps).reshape(n, H * D) * W("mix.norm") * g * torch.sigmoid(g)) @ W("mix.o").T
    if t == "latent_attention":
        rd, rank, rot = c["rot_dim"], c["kv_rank"], c["rot"]
        q = (_norm(h @ W("mix.dq").T, W("mix.dq.norm"), eps) @ W("mix.uq").T).view(n, H, D + rd)
        kv = h @ W("mix.dkv").T
        lat = _norm(kv[:, :rank], W("mix.dkv.norm"), eps)
        k, v = (lat @ W("mix.uk").T).view(n, H, D), (lat @ W("mix.uv").T).view(n, H, V)

        def one(q, k, v, kr):
            a = _angles(q.shape[0], rot["dims"], rot["base"])
            kr = _turn(kr[:, None], a, True).expand(-1, H, -1)
            return _attend(torch.cat([q[..., :D], _turn(q[..., D:], a, True)], -1), torch.cat([k, kr], -1), v, 1 << 40, c["scale"])
        o = _each(seqs, one, q, k, v, kv[:, rank:]).reshape(n, H * V)
        return (o * torch.sigmoid(h @ W("mix.g").T)) @ W("mix.o").T
    if t == "attention":
        G = c["kv_heads"]
        q = _norm(h @ W("mix.q").T + W("mix.q.b"), W("mix.q.norm"), eps).view(n, H, D)
        k = _norm(h @ W("mix.k").T + W("mix.k.b"), W("mix.k.norm"), eps).view(n, G, D)
        v = (h @ W("mix.v").T + W("mix.v.b")).view(n, G, V)
        sink, qt = W("mix.sink"), c["q_temp"]

        def one(q, k, v):
            p = torch.arange(q.shape[0], dtype=torch.float64, device=DEVICE)
            f = 1.0 + qt["coef"] * torch.log(torch.floor((p + 1) / qt["every"]) + 1.0)
            return _attend(q * f[:, None, None], k, v, 1 << 40, c["scale"], sink)
        return _each(seqs, one, q, k, v).reshape(n, H * V) @ W("mix.o").T
    decay = torch.tensor(np.array(c["decay"], dtype=np.float32), device=DEVICE).double()
    q, k, v = (h @ W("mix.q").T).view(n, H, D), (h @ W("mix.k").T).view(n, H, D), (h @ W("mix.v").T).view(n, H, V)
    g = h @ W("mix.g").T
    if t == "lightning":
        q, k, v = (x * torch.sigmoid(x) for x in (q, k, v))
        o = _each(seqs, lambda *a: _decayed(*a, decay), q, k, v).reshape(n, H * V)
        return (_norm(o, W("mix.norm"), eps) * torch.sigmoid(g)) @ W("mix.o").T
    rot = c["rot"]

    def one(q, k, v):
        a, m = _angles(q.shape[0], rot["dims"], rot["base"]), rot["dims"]
        q, k = (torch.cat([_turn(x[..., :m], a, False), x[..., m:]], -1) for x in (q, k))
        return _decayed(q, k * D ** -0.5, v, decay)
    o = _norm(_each(seqs, one, q, k, v), None, eps).reshape(n, H * V)
    return (o * g * torch.sigmoid(g)) @ W("mix.o").T


def _forward(model, layers, tokens):
    """Normed residual stream behind the last layer for every token of the sequences, stacked, in 64 bits."""
    cfg = model_config(model, layers)
    shapes = {n: (s, k) for n, s, k in weight_list(model, cfg)}

    def get(name):
        return weight(model, name, *shapes[name]).double()
    ends = np.cumsum([len(t) for t in tokens])
    seqs = [(int(e) - len(t), int(e)) for t, e in zip(tokens, ends)]
    ids = torch.from_numpy(np.concatenate(tokens).astype(np.int64)).to(DEVICE)
    name = "embed_tokens.weight" if is_gemma(model) else "embed"
    x = weight(model, name, *shapes[name])[ids].double()
    n = x.shape[0]
    if not is_gemma(model):
        eps, parallel = cfg["norm"]["eps"], cfg["architecture"] == "Nozurax"
        for i, layer in enumerate(cfg["layers"]):
            def W(name, i=i):
                return get("l%d.%s" % (i, name))
            gate, up, down = W("mlp.gate"), W("mlp.up"), W("mlp.down")
            if parallel:
                h = _norm(x, 1.0 + W("norm1"), eps)
                x = x + _mixer(layer, W, h, seqs, eps) + _rows(lambda y: (torch.relu(y @ gate.T) * (y @ up.T)) @ down.T, h)
            else:
                x = x + _norm(_mixer(layer, W, _norm(x, W("norm1"), eps), seqs, eps), W("norm1b"), eps)
                y = _rows(lambda y: (torch.nn.functional.silu(y @ gate.T) * (y @ up.T)) @ down.T, _norm(x, W("norm2"), eps))
                x = x + _norm(y, W("norm2b"), eps)
        return _norm(x, get("final.norm") + (1.0 if parallel else 0.0), eps)
    eps, H, D, Nq, Nkv = (cfg[k] for k in ("rms_norm_eps", "hidden_size", "head_dim", "num_attention_heads", "num_key_value_heads"))
    x = x * math.sqrt(H)
    for l, t in enumerate(cfg["layer_types"]):
        def W(name, l=l):
            return get("layers.%d.%s.weight" % (l, name))
        window = cfg["sliding_window"] if t == "sliding_attention" else 1 << 40
        theta = cfg["rope_parameters"][t]["rope_theta"]
        h = _norm(x, W("input_layernorm"), eps)
        q = _norm((h @ W("self_attn.q_proj").T).view(n, Nq, D), W("self_attn.q_norm"), eps)
        k = _norm((h @ W("self_attn.k_proj").T).view(n, Nkv, D), W("self_attn.k_norm"), eps)
        v = _norm((h @ W("self_attn.v_proj").T).view(n, Nkv, D), None, eps)

        def one(q, k, v):
            a = _angles(q.shape[0], D, theta)
            return _attend(_turn(q, a, False), _turn(k, a, False), v, window, 1.0)
        o = _each(seqs, one, q, k, v).reshape(n, Nq * D) @ W("self_attn.o_proj").T
        x = x + _norm(o, W("post_attention_layernorm"), eps)
        gate, up, down = W("mlp.gate_proj"), W("mlp.up_proj"), W("mlp.down_proj")
        y = _rows(lambda y: (_gelu(y @ gate.T) * (y @ up.T)) @ down.T, _norm(x, W("pre_feedforward_layernorm"), eps))
        x = x + _norm(y, W("post_feedforward_layernorm"), eps)           # layer_scalar is 1
    return _norm(x, get("norm.weight"), eps)


def _logits(model, layers, h):
    cfg = model_config(model, layers)
    V, H = vocab_of(model, cfg), h.shape[1]
    w = weight(model, "embed_tokens.weight" if is_gemma(model) else "head", (V, H), "matrix")
    return torch.cat([h @ w[i:i + 32768].double().T for i in range(0, V, 32768)], 1)


def exact(case, seed):
    model, layers, steps = case["model"], case["layers"], case["steps"]
    if work(case)["flops"] > 3e14:               # about ten seconds of 64-bit arithmetic
        return None
    cfg = model_config(model, layers)
    prompts = [p.astype(np.int64) for p in _prompts(case, cfg, seed)]

    def walk(token, count):                      # the tokens that follow by the clear margin
        out = []
        for _ in range(count):
            token = int(successor(model, cfg, token))
            out.append(token)
        return out
    if case["call"] == "turns":
        seq, places, at = [], [], 0
        for n in portions(case):
            seq += list(prompts[0][at:at + n])
            at += n
            # the answer's tokens follow each other; the last one's successor is not fed
            answer = walk(seq[-1], steps)
            places += list(range(len(seq) - 1, len(seq) + steps))
            seq += answer
        h = _forward(model, layers, [np.array(seq)])[places]
        return {"logits": _logits(model, layers, h)}
    # tokens fed behind the prompt: serve starts from the last prompt token, the others from its successor
    fed = [walk(p[-1], steps + (case["call"] == "greedy")) for p in prompts]
    seqs = [np.concatenate([p, np.array(f, dtype=np.int64)]) for p, f in zip(prompts, fed)]
    h = _forward(model, layers, seqs)
    ends = np.cumsum([len(s) for s in seqs])
    last = _logits(model, layers, h[[int(e) - 1 for e in ends]]) if case["call"] != "topk" else None
    if case["call"] == "serve":
        return {"ids": None, "last": last}
    head = _logits(model, layers, h[[int(e) - len(s) + len(p) - 1 for e, s, p in zip(ends, seqs, prompts)]])
    head = head[0] if case["batch"] == 1 else head
    if case["call"] == "greedy":
        return {"logits": head, "ids": None, "last": last[0] if case["batch"] == 1 else last}
    scores = []
    for i in range(steps):
        row = _logits(model, layers, h[len(prompts[0]) + i][None])[0]
        seen = torch.tensor(sorted(set(fed[0][:i + 1])), device=DEVICE)
        row[seen] = torch.where(row[seen] >= 0, row[seen] / float(np.float32(1.1)), row[seen] * float(np.float32(1.1)))
        scores.append(torch.topk(row, 40).values)
    return {"logits": head, "ids": None, "scores": torch.stack(scores)}
