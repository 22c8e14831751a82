"""The work whose speed this framework is judged by: decode steps at batch 1, batched decode steps and prompts
prefilled in chunks, through the engines a program calls (`DecodeEngine`, `BatchDecodeEngine`, `PrefillEngine`).

A case is one engine configuration at one context length.  Widths are those of the repository's named
configurations (8B Llama and Qwen3 shapes, the 30B mixture of experts) and of its tests; most cases hold a few layers
of them, so that the outputs (hidden states, logits, cache rows) say something about each layer's arithmetic, and
enough weight bytes that a pass does not find them in L2.
"""
import math

import torch

BF16 = torch.bfloat16
PAGE, D = 64, 128
DEV = "cuda:0"

LLAMA_8B = dict(hidden=4096, heads=32, kv=8, ffn=14336, eps=1e-5, theta=5e5, qk_norm=False)
QWEN3_8B = dict(hidden=4096, heads=32, kv=8, ffn=12288, eps=1e-6, theta=1e6, qk_norm=True)
QWEN3_MOE = dict(hidden=2048, heads=32, kv=4, ffn=768, eps=1e-6, theta=1e6, qk_norm=True, experts=128, top_k=8)
SMALL = dict(hidden=512, heads=8, kv=2, ffn=1024, eps=1e-5, theta=5e5, qk_norm=False)


def _case(path, shape, layers, vocab, ctx, fmt="bf16", batch=1, chunk=0, name=None):
    c = dict(path=path, layers=layers, vocab=vocab, ctx=ctx, fmt=fmt, batch=batch, chunk=chunk, experts=0, top_k=0)
    c.update(shape)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # one token of a small model (the tests' shape): launch, stage and host latency
        _case("decode", SMALL, 3, 2048, 199, name="decode_small"),
        # one token of an 8B model after the benchmark's prompt, with the whole vocabulary projection and its logits
        _case("decode", LLAMA_8B, 8, 128256, 2112, name="decode_8b"),
        # the same model's layers with FP8 rows, at a short ragged context (a chat's first turns)
        _case("decode", LLAMA_8B, 4, 16384, 333, fmt="fp8", name="decode_8b_fp8"),
        # NVFP4 rows with q/k norms after a 4096-token prompt
        _case("decode", QWEN3_8B, 4, 16384, 4131, fmt="nvfp4", name="decode_8b_nvfp4"),
        # one token through mixture-of-experts layers
        _case("decode", QWEN3_MOE, 4, 16384, 2050, name="decode_moe"),
        # a handful of sequences, e.g. parallel samples of one request
        _case("batch", LLAMA_8B, 2, 16384, 1000, batch=3, name="batch3"),
        # serving batches: ordinary, quantised, large; every sequence at a length of its own
        _case("batch", QWEN3_8B, 2, 16384, 4100, fmt="nvfp4", batch=16, name="batch16_nvfp4"),
        _case("batch", LLAMA_8B, 2, 16384, 1500, fmt="fp8", batch=32, name="batch32_fp8"),
        _case("batch", LLAMA_8B, 2, 32768, 2100, batch=64, name="batch64"),
        _case("batch", LLAMA_8B, 2, 16384, 700, batch=128, name="batch128"),
        # a short ragged prompt (one and a bit chunks), and the benchmark's prompt length
        _case("prefill", QWEN3_8B, 2, 16384, 77, chunk=64, name="prefill_77"),
        _case("prefill", LLAMA_8B, 2, 16384, 2048, chunk=128, name="prefill_2048"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    path = rng.choice(["decode", "decode", "batch", "batch", "batch", "prefill"])
    fmt = rng.choice(["bf16", "bf16", "fp8", "nvfp4"])
    base = dict(rng.choice([LLAMA_8B, QWEN3_8B, LLAMA_8B, SMALL]))
    if base["hidden"] == 512 and fmt == "nvfp4":
        base["hidden"] = 1024       # NVFP4 rows come in multiples of 1024 inputs
    if rng.random() < 0.3:          # other widths of the same kind
        base["hidden"] = 1024 * rng.randint(1, 4)
        base["ffn"] = 1024 * rng.randint(1, 14)
        base["kv"] = rng.choice([1, 2, 4, 8])
        base["heads"] = base["kv"] * rng.choice([4, 8])
        while base["heads"] * D % 1024:
            base["heads"] *= 2
            base["kv"] *= 2
    vocab = 256 * rng.randint(4, 64)
    if path == "decode":
        if fmt == "bf16" and rng.random() < 0.2:
            return _case("decode", QWEN3_MOE, rng.randint(1, 4), vocab, _log(rng, 1, 4000))
        return _case("decode", base, rng.randint(1, 4), vocab, _log(rng, 1, 8000), fmt)
    if path == "batch":
        b = _log(rng, 2, 128)
        return _case("batch", base, rng.randint(1, 2), vocab, _log(rng, 1, min(4200, 131072 // b)), fmt, batch=b)
    return _case("prefill", base, rng.randint(1, 2), vocab, _log(rng, 2, 1500), fmt, chunk=rng.choice([32, 64, 128, 128]))


# ------------------------------------------------------------------ inputs
def _rng(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


def _matrix(g, m, k, fmt, std=0.02):
    """[m, k] bf16 weights.  For the quantised formats they lie on the format's grid (e4m3 codes under a row scale;
    e2m1 codes under block scales), as weights read back from a quantised checkpoint do."""
    x = torch.empty(m, k, device=DEV).normal_(generator=g)
    if fmt == "fp8":
        x = (x * 82).clamp_(-448, 448)
        x[:, 0] = 448.0
        return (x.to(torch.float8_e4m3fn).float() * 2.0 ** -12).to(BF16)
    if fmt == "nvfp4":
        grid = torch.tensor([0.0, 0.5, 1.0, 1.5, 2.0, 3.0, 4.0, 6.0], device=DEV)
        mids = (grid[1:] + grid[:-1]) / 2
        v = (grid[torch.bucketize(x.abs() * 2, mids)] * x.sign()).view(m, k // 16, 16)
        v[:, :, 0] = 6.0
        s = 256.0 + 64.0 * torch.randint(0, 4, (m, k // 16, 1), generator=g, device=DEV)
        s[0, 0] = 448.0
        return (v * s * 2.0 ** -15).view(m, k).to(BF16)
    return (x * std).to(BF16)


def _weights(c, seed):
    """A model's weights as lists with one entry per layer."""
    g = _rng(seed)
    H, F, q, kv, fmt = c["hidden"], c["ffn"], c["heads"] * D, c["kv"] * D, c["fmt"]
    near = lambda n, at=1.0: (at * (1 + 0.1 * torch.empty(n, device=DEV).normal_(generator=g))).to(BF16)
    w = {k: [] for k in ("ln1", "ln2", "wq", "wk", "wv", "wo", "gate", "up", "down", "router", "q_norm", "k_norm")}
    w["embed"] = (torch.empty(c["vocab"], H, device=DEV).normal_(generator=g) * 0.5).to(BF16)
    w["lm_head"] = _matrix(g, c["vocab"], H, "bf16")
    w["norm"] = near(H)
    for _ in range(c["layers"]):
        w["ln1"].append(near(H))
        w["ln2"].append(near(H))
        w["wq"].append(_matrix(g, q, H, fmt))
        w["wk"].append(_matrix(g, kv, H, fmt))
        w["wv"].append(_matrix(g, kv, H, fmt))
        w["wo"].append(_matrix(g, H, q, fmt))
        if c["qk_norm"]:
            w["q_norm"].append(near(D, 1.5))
            w["k_norm"].append(near(D, 1.5))
        if c["experts"]:
            w["gate"].append([_matrix(g, F, H, fmt) for _ in range(c["experts"])])
            w["up"].append([_matrix(g, F, H, fmt) for _ in range(c["experts"])])
            w["down"].append([_matrix(g, H, F, fmt) for _ in range(c["experts"])])
            w["router"].append(_matrix(g, c["experts"], H, "bf16", 0.08))
        else:
            w["gate"].append(_matrix(g, F, H, fmt))
            w["up"].append(_matrix(g, F, H, fmt))
            w["down"].append(_matrix(g, H, F, fmt))
    return w


def _contexts(c):
    """Cached positions of each sequence: one at the case's context, the others between half of it and all of it."""
    return [c["ctx"] - (b * 37) % max(1, c["ctx"] // 2) for b in range(c["batch"])]


def _cache(c, seed, b):
    """Sequence b's cached key and value rows, per layer [T, kv heads, 128]."""
    g = _rng(seed * 1000 + b + 1)
    T = _contexts(c)[b]
    rows = lambda: torch.empty(c["layers"], T, c["kv"], D, device=DEV, dtype=BF16).normal_(generator=g)
    return rows(), rows()


def _tokens(c, seed):
    n = c["ctx"] if c["path"] == "prefill" else c["batch"]
    return torch.randint(0, c["vocab"], (n,), generator=torch.Generator().manual_seed(seed))


def prepare(case, seed):
    from vdcores_b200.batch import BatchDecodeEngine
    from vdcores_b200.decode import DecodeConfig, DecodeEngine, DenseWeights
    from vdcores_b200.prefill import PrefillEngine
    c = case
    cfg = DecodeConfig(hidden=c["hidden"], n_heads=c["heads"], n_kv_heads=c["kv"], head_dim=D, ffn=c["ffn"],
                       vocab=c["vocab"], n_layers=c["layers"], eps=c["eps"], theta=c["theta"], qk_norm=c["qk_norm"],
                       n_experts=c["experts"], top_k=c["top_k"] or 8)
    max_seq = (c["ctx"] + 256) // PAGE * PAGE
    if c["path"] == "batch":
        e = BatchDecodeEngine(cfg, c["batch"], max_seq, device=DEV, wkind=c["fmt"])
    else:
        e = DecodeEngine(cfg, max_seq, device=DEV, wkind=c["fmt"])
    w = _weights(c, seed)
    e.load_weights(DenseWeights(**{k: (v if len(v) else None) for k, v in w.items()}))
    tokens = _tokens(c, seed)
    s = dict(case=c, engine=e, tokens=tokens)
    if c["path"] == "prefill":
        s["prefill"] = PrefillEngine(e, chunk=c["chunk"]).adopt_weights()
        return s
    for b, T in enumerate(_contexts(c)):
        k, v = _cache(c, seed, b)
        if c["path"] == "batch":
            e.load_kv(list(k), list(v), b=b)
            torch.cuda.synchronize()        # the state block goes up from one pinned buffer
            e.set_state(T, int(tokens[b]), b=b)
        else:
            e.load_kv(list(k), list(v))
            e.set_state(T, int(tokens[b]))
    torch.cuda.synchronize()
    s["state"], s["pos"] = e.state.clone(), e.pos
    return s


def run(state):
    """A decode step from the state's position, or a whole prompt."""
    e = state["engine"]
    if "prefill" in state:
        p = state["prefill"]
        p.prefill(state["tokens"])
        return {"hidden": p.read_hidden(p.hidden), "k": e.kpool, "v": e.vpool}
    e.state.copy_(state["state"])       # the step moves its state block on: take it back to the same position
    e.pos, e.steps_done = state["pos"], 0
    e.step_async()
    if state["case"]["path"] == "batch":
        return {"hidden": e.read_hidden(e.hidden)}
    return {"hidden": e.hidden, "logits": e.logits}


def work(case):
    c = case
    H, F, q, kv, L = c["hidden"], c["ffn"], c["heads"] * D, c["kv"] * D, c["layers"]
    attn = H * (q + 2 * kv) + q * H
    ffn = 3 * H * F * (c["top_k"] if c["experts"] else 1)
    per = {"bf16": 2.0, "fp8": 1.0, "nvfp4": 9 / 16}[c["fmt"]]
    n = c["ctx"] if c["path"] == "prefill" else c["batch"]
    bytes_ = L * ((attn + ffn) * per + c["experts"] * H * 2) + c["vocab"] * H * 2 + n * H * 2
    flops = 2.0 * n * L * (attn + ffn + c["experts"] * H)
    if c["path"] == "prefill":
        bytes_ += 2 * 2 * kv * n * L
        flops += 2.0 * c["vocab"] * H + 4.0 * q * L * n * (n + 1) / 2
    else:
        ctxs = [t + 1 for t in _contexts(c)]
        bytes_ += 2 * 2 * kv * sum(ctxs) * L
        flops += 2.0 * n * c["vocab"] * H + 4.0 * q * L * sum(ctxs)
    return {"bytes": bytes_, "flops": flops}


def tolerance(case):
    """bf16 activations between the stages of a layer: against 64 bits the outputs are 0.3e-2 (small, norms on the heads)
    to 1.9e-2 off (eight layers, or a second layer's hidden states after few positions), and the same step with its fp32
    sums in another order is up to 0.8e-2 from itself.  Two correct orders of rounding differ by about the larger of
    the errors times the square root of two."""
    return {"rel": 3e-2}


# ------------------------------------------------------------------ the same in 64 bits
def exact(case, seed):
    c = case
    w, tokens = _weights(c, seed), _tokens(c, seed)
    H, hq, hk, L = c["hidden"], c["heads"], c["kv"], c["layers"]
    f64 = lambda t: t.double()
    norm = lambda x, g, eps: x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + eps) * f64(g)
    inv = 1.0 / (c["theta"] ** (torch.arange(0, D, 2, dtype=torch.float32) / D))

    def rope(x, pos):       # [n, heads, 128]; the angles' sines and cosines are bf16 tables
        fr = pos.float().cpu()[:, None] * inv[None, :]
        cos, sin = (t.to(BF16).double().to(DEV)[:, None, :] for t in (fr.cos(), fr.sin()))
        a, b = x[..., :64], x[..., 64:]
        return torch.cat((a * cos - b * sin, b * cos + a * sin), -1)

    prefill = c["path"] == "prefill"
    pos = torch.arange(c["ctx"]) if prefill else torch.tensor(_contexts(c))
    caches = None if prefill else [_cache(c, seed, b) for b in range(c["batch"])]
    h = f64(w["embed"][tokens.to(DEV)])
    n = h.shape[0]
    new_k, new_v = [], []
    for l in range(L):
        x = norm(h, w["ln1"][l], c["eps"])
        qh, kh, vh = ((x @ f64(w[m][l]).t()).view(n, -1, D) for m in ("wq", "wk", "wv"))
        if c["qk_norm"]:
            qh, kh = norm(qh, w["q_norm"][l], 1e-6), norm(kh, w["k_norm"][l], 1e-6)
        qh, kh = rope(qh, pos), rope(kh, pos)
        new_k.append(kh)
        new_v.append(vh)
        o = torch.empty(n, hq, D, dtype=torch.float64, device=DEV)
        G = hq // hk
        if prefill:
            mask = torch.ones(n, n, dtype=torch.bool, device=DEV).triu(1)
            for i in range(hq):
                sc = (qh[:, i] @ kh[:, i // G].t() / math.sqrt(D)).masked_fill(mask, -math.inf)
                o[:, i] = torch.softmax(sc, -1) @ vh[:, i // G]
        else:
            for b in range(n):
                ck, cv = caches[b]
                K, V = torch.cat((f64(ck[l]), kh[b:b + 1])), torch.cat((f64(cv[l]), vh[b:b + 1]))
                sc = torch.einsum("kgd,tkd->kgt", qh[b].view(hk, G, D), K) / math.sqrt(D)
                o[b] = torch.einsum("kgt,tkd->kgd", torch.softmax(sc, -1), V).reshape(hq, D)
        h = h + o.view(n, -1) @ f64(w["wo"][l]).t()
        x = norm(h, w["ln2"][l], c["eps"])
        ffn = lambda x, g, u, d: (torch.nn.functional.silu(x @ f64(g).t()) * (x @ f64(u).t())) @ f64(d).t()
        if c["experts"]:
            p, ids = torch.softmax(x @ f64(w["router"][l]).t(), -1).topk(c["top_k"], -1)
            p = p / p.sum(-1, keepdim=True)
            h = h + torch.stack([sum(p[b, j] * ffn(x[b], *(w[m][l][int(ids[b, j])] for m in ("gate", "up", "down")))
                                     for j in range(c["top_k"])) for b in range(n)])
        else:
            h = h + ffn(x, w["gate"][l], w["up"][l], w["down"][l])
    if c["path"] == "batch":
        return {"hidden": h}
    if not prefill:
        return {"hidden": h[0], "logits": f64(w["lm_head"]) @ norm(h, w["norm"], c["eps"])[0]}
    # cache pages as they lie in the pools: [layer, page, kv head, 64 rows, 128], the 16-byte pieces of a row at
    # (piece XOR row mod 8); the last chunk's rows past the prompt repeat its last position
    pages = ((c["ctx"] + 256) // PAGE * PAGE + PAGE - 1) // PAGE
    row = torch.arange(PAGE, device=DEV)
    piece = torch.arange(D // 8, device=DEV)[None, :] ^ (row[:, None] & 7)

    def pool(rows):
        t = torch.zeros(L, pages * PAGE, hk, D, dtype=torch.float64, device=DEV)
        t[:, :n] = torch.stack(rows)
        t = t.view(L, pages, PAGE, hk, D // 8, 8).transpose(2, 3)
        return t[:, :, :, row[:, None], piece].reshape(L, pages, hk, PAGE, D)

    B = c["chunk"]
    last = torch.arange((n - 1) // B * B, (n - 1) // B * B + B, device=DEV).clamp_(max=n - 1)
    return {"hidden": h[last], "k": pool(new_k), "v": pool(new_v)}
