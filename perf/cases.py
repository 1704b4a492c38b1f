"""The work that programs built on this package have it do, as timed cases over ranges of sizes.

Sequence-state decoders (umbrella_b200.ops_seq, models.zedotar): the matrix products of a step, the routed experts, cached
attention in prompts and in decode steps, attention over per-head keys of a prompt, the retention recurrence, and a whole
served batch.  Speculative decoding (models.llama): a token tree verified by an INT4 target, and a prompt.

``listed()`` and ``draw(rng)`` give cases (plain dicts); ``prepare`` makes what a program holds before the call, ``run`` is
one pass through the public entry points, ``work`` what the pass cannot do without, ``exact`` the same result in 64 bits from
plain torch, ``tolerance`` how far a correct implementation at the same precision may be from another.
"""
import math

import torch

DEV = "cuda:0"
F64 = torch.float64


def listed():
    return [
        # the in-projection of a width-2048 layer in a decode step of eight sequences
        dict(name="linear_decode", kind="linear", rows=8, k=2048, n=6144, dtype="bf16", f32_out=True),
        # the same product over a prompt's tokens
        dict(name="linear_prompt", kind="linear", rows=4096, k=2048, n=6144, dtype="bf16", f32_out=True),
        # a model served in true 32-bit: an odd number of rows, the in-projection of a width-1024 matrix-memory layer
        dict(name="linear_fp32", kind="linear", rows=777, k=1024, n=3088, dtype="f32", f32_out=True),
        # the routed feed-forward of a decode step of 64 sequences, and of a prompt
        dict(name="experts_decode", kind="experts", tokens=64, width=2048, experts=16, top=2, ff=1024),
        dict(name="experts_prompt", kind="experts", tokens=4096, width=2048, experts=16, top=2, ff=1024),
        # grouped-query attention with a window, pooled blocks behind it and a sink: 64 sequences decoding, one long prompt
        dict(name="attention_decode", kind="attention", seqs=64, tokens=1, context=2000, heads=16, kv_heads=4, dim=128, window=1024, pool=64),
        dict(name="attention_prompt", kind="attention", seqs=1, tokens=4096, context=0, heads=16, kv_heads=4, dim=128, window=1024, pool=64),
        # two unequal fresh prompts through latent attention's per-head form: shared rotated key part, sink, output gate
        dict(name="latent_prompt", kind="latent", seqs=2, tokens=2000, heads=16, dim=128, shared=64, vdim=128, window=0),
        # the decayed linear-attention recurrence over a prompt
        dict(name="retention_prompt", kind="retention", seqs=1, tokens=4096, heads=16, dim=64, vdim=128),
        # a 13-node token tree verified behind 512 tokens by one layer and the head of the 70B INT4 target
        dict(name="verify_tree", kind="llama", size="70b", tokens=13, prefix=512, tree=True),
        # a prompt of ordinary length through one layer and the head of the 8B INT4 draft
        dict(name="draft_prompt", kind="llama", size="8b", tokens=500, prefix=0, tree=False),
        # four requests served by the batch engine's model: one ragged prompt step, then decode steps
        dict(name="served_batch", kind="served", width=1024, layers=8, seqs=4, tokens=256, steps=8),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["linear", "linear", "linear", "experts", "experts", "attention", "attention", "latent", "retention", "llama",
                       "llama", "served"])
    if kind == "linear":
        if rng.random() < 0.25:
            return dict(kind=kind, rows=_log(rng, 1, 800), k=rng.choice([512, 1000, 1024]), n=rng.choice([513, 1024, 3088]), dtype="f32",
                        f32_out=True)
        k = rng.choice([384, 768, 1024, 1536, 2048, 4096])
        n = rng.choice([250, 512, 1024, 1544, 2048, 3088, 4096, 6144])
        return dict(kind=kind, rows=_log(rng, 1, 4096), k=k, n=n, dtype="bf16", f32_out=rng.random() < 0.5)
    if kind == "experts":
        width = rng.choice([1024, 2048])
        return dict(kind=kind, tokens=_log(rng, 1, 4096), width=width, experts=rng.choice([8, 16]), top=rng.choice([1, 2, 4])
                    if width == 1024 else 2, ff=width // 2)
    if kind == "attention":
        heads = rng.choice([8, 16])
        shape = dict(kind=kind, heads=heads, kv_heads=rng.choice([2, 4, heads]), dim=rng.choice([64, 96, 128]))
        window, pool = rng.choice([(0, 0), (512, 0), (1024, 64)])
        if rng.random() < 0.5:
            return dict(shape, seqs=_log(rng, 1, 64), tokens=1, context=_log(rng, 1, 2000), window=window, pool=pool)
        # a prompt, or a later portion of one
        return dict(shape, seqs=rng.choice([1, 2, 3]), tokens=_log(rng, 16, 1300), context=rng.choice([0, 0, 700]), window=window, pool=pool)
    if kind == "latent":
        return dict(kind=kind, seqs=rng.choice([1, 2, 4]), tokens=_log(rng, 16, 1500), heads=rng.choice([8, 16]), dim=rng.choice([64, 128]),
                    shared=rng.choice([0, 32, 64]), vdim=rng.choice([64, 128]), window=rng.choice([0, 0, 700]))
    if kind == "retention":
        return dict(kind=kind, seqs=rng.choice([1, 2, 8]), tokens=_log(rng, 1, 512), heads=rng.choice([8, 16]), dim=64,
                    vdim=rng.choice([64, 128]))
    if kind == "llama":
        if rng.random() < 0.6:
            return dict(kind=kind, size=rng.choice(["8b", "70b"]), tokens=_log(rng, 1, 64), prefix=_log(rng, 16, 3000), tree=True)
        return dict(kind=kind, size="8b", tokens=_log(rng, 16, 1000), prefix=0, tree=False)
    return dict(kind=kind, width=rng.choice([512, 1024]), layers=rng.choice([4, 8]), seqs=_log(rng, 1, 16), tokens=_log(rng, 16, 256),
                steps=rng.choice([4, 8]))


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


def _randn(g, *shape, scale=1.0, dtype=torch.float32):
    return (torch.randn(shape, generator=g, device=DEV) * scale).to(dtype)


def _lengths(case):
    """Ragged steps: the first sequence is the longest, each further one about a seventh shorter than the one before it."""
    return [max(1, int(case["tokens"] * (1 - i / 7))) if i < 6 else max(1, case["tokens"] // 7) for i in range(case["seqs"])]


def _starts(case):
    """Tokens every sequence has behind it: the case's context, a little less for each further sequence."""
    return [max(0, case["context"] - 3 * i) for i in range(case["seqs"])]


# ---------------------------------------------------------------------------------------------- matrix product
def _linear_inputs(c, seed):
    g, dt = _gen(seed), torch.bfloat16 if c["dtype"] == "bf16" else torch.float32
    return _randn(g, c["rows"], c["k"], dtype=dt), _randn(g, c["n"], c["k"], scale=c["k"] ** -0.5, dtype=dt)


def _linear_prepare(c, seed):
    a, w = _linear_inputs(c, seed)
    return dict(a=a, w=w)


def _linear_run(c, s):
    from umbrella_b200 import ops_seq
    return ops_seq.gemm(s["a"], s["w"], out_f32=c["f32_out"])


def _linear_exact(c, seed):
    a, w = _linear_inputs(c, seed)
    return a.to(F64) @ w.to(F64).T


def _linear_work(c):
    e = 2 if c["dtype"] == "bf16" else 4
    return dict(bytes=e * c["k"] * (c["rows"] + c["n"]) + (4 if c["f32_out"] else e) * c["rows"] * c["n"], flops=2 * c["rows"] * c["k"] * c["n"])


# ---------------------------------------------------------------------------------------------- routed experts
_LIMIT, _EPS = 7.0, 1e-6


def _experts_inputs(c, seed):
    g, W, E, ff, bf = _gen(seed), c["width"], c["experts"], c["ff"], torch.bfloat16
    return dict(h=_randn(g, c["tokens"], W, dtype=bf), x=_randn(g, c["tokens"], W), router=_randn(g, E, W, scale=W ** -0.5),
                gu=_randn(g, E, 2 * ff, W, scale=W ** -0.5, dtype=bf), down=_randn(g, E, W, ff, scale=ff ** -0.5, dtype=bf),
                norm=1 + _randn(g, W, scale=0.1))


def _experts_prepare(c, seed):
    s = _experts_inputs(c, seed)
    s["rows"] = torch.arange(c["tokens"], dtype=torch.int32, device=DEV)
    return s


def _experts_run(c, s):
    """Route, gate|up with the activation, down, then the weighted sum, the residual and the next norm."""
    from umbrella_b200 import _lib_seq, ops_seq
    n, top = c["tokens"], c["top"]
    sel_w, grp_off, pair_tok, pair_pos, _ = ops_seq.moe_route(s["h"], s["router"], top)
    y = ops_seq.gemm(s["h"], s["gu"], groups=c["experts"], n=c["ff"], dual=True, limit=_LIMIT, grp_off=grp_off, row_src=pair_tok,
                     rows=n * top, max_rows=n)
    o = ops_seq.gemm(y, s["down"], out_f32=True, groups=c["experts"], grp_off=grp_off, rows=n * top, max_rows=n)
    return ops_seq.add_norm(s["x"], s["norm"], None, _EPS, kind=_lib_seq.UMBS_NORM_RMS, dtype=torch.bfloat16, rows=s["rows"], pair_out=o,
                            sel_w=sel_w, pair_pos=pair_pos, want_copy=True)


def _experts_exact(c, seed):
    s = _experts_inputs(c, seed)
    h, ff = s["h"].to(F64), c["ff"]
    val, idx = torch.topk(h @ s["router"].to(F64).T, c["top"], dim=-1)
    p = torch.softmax(val, -1)
    x = s["x"].to(F64)
    for e in range(c["experts"]):
        tok, which = torch.nonzero(idx == e, as_tuple=True)
        if tok.numel():
            w = s["gu"][e].to(F64)
            gate, up = (h[tok] @ w[:ff].T).clamp(max=_LIMIT), (h[tok] @ w[ff:].T).clamp(-_LIMIT, _LIMIT)
            out = (gate * torch.sigmoid(1.702 * gate) * (up + 1)) @ s["down"][e].to(F64).T
            x.index_add_(0, tok, p[tok, which, None] * out)
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + _EPS) * s["norm"].to(F64), x


def _experts_work(c):
    n, W, ff, top = c["tokens"], c["width"], c["ff"], c["top"]
    touched = min(c["experts"], n * top)
    return dict(bytes=touched * 3 * ff * W * 2 + c["experts"] * W * 4 + n * W * (2 + 4 + 2 + 4), flops=2 * n * top * 3 * ff * W)


# ---------------------------------------------------------------------------------------------- attention over a cache
def _attention_inputs(c, seed):
    g, bf = _gen(seed), torch.bfloat16
    row = c["kv_heads"] * 2 * c["dim"]
    lens, pos = _lengths(c), _starts(c)
    cap = max(n + p for n, p in zip(lens, pos))
    return dict(q=_randn(g, sum(lens), c["heads"] * c["dim"], dtype=bf), kv=_randn(g, sum(lens), row, dtype=bf),
                cache=_randn(g, c["seqs"], cap, row, dtype=bf), sink=_randn(g, c["heads"]), gate=_randn(g, sum(lens), c["heads"]))


def _attention_prepare(c, seed):
    from umbrella_b200 import ops_seq
    s = _attention_inputs(c, seed)
    lens, pos, cap = _lengths(c), _starts(c), s["cache"].shape[1]
    if c["pool"]:
        # what earlier steps left: the mean row of every block of older tokens
        blocks = -(-cap // c["pool"])
        s["pools"] = torch.zeros(c["seqs"], blocks, s["cache"].shape[2], dtype=torch.bfloat16, device=DEV)
        full = cap // c["pool"]
        s["pools"][:, :full] = s["cache"][:, :full * c["pool"]].float().reshape(c["seqs"], full, c["pool"], -1).mean(2).to(torch.bfloat16)
    s["batch"] = ops_seq.RaggedBatch([(i, n, p, 0) for i, (n, p) in enumerate(zip(lens, pos))], DEV)
    return s


def _attention_run(c, s):
    from umbrella_b200 import _lib_seq, ops_seq
    out = ops_seq.cached_attention(s["q"], s["kv"], s["cache"], s["batch"], c["heads"], c["kv_heads"], c["dim"], c["dim"], c["dim"] ** -0.5,
                                   mode=_lib_seq.UMBS_ATTN_SOFTMAX_SINK, window=c["window"], pool=c["pool"], pool_cache=s.get("pools"),
                                   gate=s["gate"], gate_per_head=True, sink=s["sink"])
    return (out, s["cache"], s["pools"]) if c["pool"] else (out, s["cache"])


def _softmax_rows(q, k, v, mask, scale, sink):
    """One head: q [n, d], k [m, d], v [m, e], mask [n, m], sink a score without a value (or None)."""
    z = (q @ k.T * scale).masked_fill(~mask, -math.inf)
    m = z.max(-1, keepdim=True).values
    if sink is not None:
        m = m.clamp(min=float(sink))
    p = torch.exp(z - m)
    return (p @ v) / (p.sum(-1, keepdim=True) + (torch.exp(sink - m) if sink is not None else 0))


def _attention_exact(c, seed):
    s = _attention_inputs(c, seed)
    H, G, D, at = c["heads"], c["kv_heads"], c["dim"], 0
    out = torch.empty(s["q"].shape[0], H, D, dtype=F64, device=DEV)
    for i, (n, p0) in enumerate(zip(_lengths(c), _starts(c))):
        rows = torch.cat([s["cache"][i, :p0], s["kv"][at:at + n]]).to(F64)
        k, v = rows[:, :G * D].reshape(-1, G, D), rows[:, G * D:].reshape(-1, G, D)
        pos, j = torch.arange(p0, p0 + n, device=DEV)[:, None], torch.arange(p0 + n, device=DEV)[None]
        mask = (j <= pos) & (j > pos - (c["window"] or 1 << 30))
        if c["pool"] and (p0 + n) // c["pool"]:
            nb = (p0 + n) // c["pool"]
            mean = lambda t: t[:nb * c["pool"]].reshape(nb, c["pool"], G, D).mean(1)
            k, v = torch.cat([mean(k), k]), torch.cat([mean(v), v])
            mask = torch.cat([(torch.arange(nb, device=DEV)[None] + 1) * c["pool"] <= pos - c["window"] + 1, mask], 1)
        q = s["q"][at:at + n].to(F64).reshape(n, H, D)
        for h in range(H):
            g = h // (H // G)
            out[at:at + n, h] = _softmax_rows(q[:, h], k[:, g], v[:, g], mask, D ** -0.5, s["sink"][h].to(F64))
        at += n
    out *= torch.sigmoid(s["gate"].to(F64))[:, :, None]
    return (out.reshape(at, H * D), None, None) if c["pool"] else (out.reshape(at, H * D), None)


def _attention_work(c):
    D, row = c["dim"], c["kv_heads"] * 2 * c["dim"]
    window, pairs, read = c["window"] or 1 << 30, 0, 0
    for n, p0 in zip(_lengths(c), _starts(c)):
        seen = [min(p + 1, window) + (max(0, p - window + 1) // c["pool"] if c["pool"] else 0) for p in (p0, p0 + n - 1)]
        # keys seen per row grow evenly up to the window and (pooled) more slowly behind it
        full = min(max(window - p0, 0), n)
        pairs += full * (seen[0] + min(p0 + full, window)) // 2 + (n - full) * ((window if full else seen[0]) + seen[1]) // 2
        read += min(p0, window) + (max(0, p0 - window) // c["pool"] if c["pool"] else 0)
    n = sum(_lengths(c))
    return dict(bytes=2 * (read * row + n * (2 * row + 2 * c["heads"] * D)), flops=4 * pairs * c["heads"] * D)


# ---------------------------------------------------------------------------------------------- attention of fresh prompts
def _latent_inputs(c, seed):
    g, bf, n = _gen(seed), torch.bfloat16, sum(_lengths(c))
    H = c["heads"]
    return dict(q=_randn(g, n, H * (c["dim"] + c["shared"]), dtype=bf), kv=_randn(g, n, H * (c["dim"] + c["vdim"]), dtype=bf),
                ks=_randn(g, n, c["shared"], dtype=bf) if c["shared"] else None, sink=_randn(g, H), gate=_randn(g, n, H * c["vdim"]))


def _latent_prepare(c, seed):
    from umbrella_b200 import ops_seq
    s = _latent_inputs(c, seed)
    s["batch"] = ops_seq.RaggedBatch([(i, n, 0, 0) for i, n in enumerate(_lengths(c))], DEV)
    return s


def _latent_run(c, s):
    from umbrella_b200 import ops_seq
    hd = c["heads"] * c["dim"]
    return ops_seq.window_attention_shared(s["q"], s["kv"][:, :hd], s["ks"], s["kv"][:, hd:], s["batch"], c["heads"],
                                           (c["dim"] + c["shared"]) ** -0.5, window=c["window"], sink=s["sink"], gate=s["gate"])


def _latent_exact(c, seed):
    s = _latent_inputs(c, seed)
    H, D, R, V, at = c["heads"], c["dim"], c["shared"], c["vdim"], 0
    out = torch.empty(s["q"].shape[0], H, V, dtype=F64, device=DEV)
    for n in _lengths(c):
        q = s["q"][at:at + n].to(F64).reshape(n, H, D + R)
        k, v = s["kv"][at:at + n, :H * D].to(F64).reshape(n, H, D), s["kv"][at:at + n, H * D:].to(F64).reshape(n, H, V)
        i = torch.arange(n, device=DEV)
        mask = (i[None] <= i[:, None]) & (i[None] > i[:, None] - (c["window"] or 1 << 30))
        for h in range(H):
            key = torch.cat([k[:, h], s["ks"][at:at + n].to(F64)], 1) if R else k[:, h]
            out[at:at + n, h] = _softmax_rows(q[:, h], key, v[:, h], mask, (D + R) ** -0.5, s["sink"][h].to(F64))
        at += n
    return out.reshape(at, H * V) * torch.sigmoid(s["gate"].to(F64))


def _latent_work(c):
    H, n = c["heads"], sum(_lengths(c))
    w = c["window"] or 1 << 30
    pairs = sum(m * (m + 1) // 2 if m <= w else w * (w + 1) // 2 + (m - w) * w for m in _lengths(c))
    return dict(bytes=2 * n * (H * (2 * c["dim"] + c["shared"] + 2 * c["vdim"]) + c["shared"]) + 4 * n * H * c["vdim"],
                flops=2 * pairs * H * (c["dim"] + c["shared"] + c["vdim"]))


# ---------------------------------------------------------------------------------------------- retention
def _retention_inputs(c, seed):
    g, H = _gen(seed), c["heads"]
    decay = torch.tensor([1 - 2.0 ** (-5 - (3 * h) // H) for h in range(H)], device=DEV)
    freq = (1e6 ** (-torch.arange(0, c["dim"], 2, dtype=F64, device=DEV) / c["dim"])).float()
    return dict(x=_randn(g, sum(_lengths(c)), 2 * H * (c["dim"] + c["vdim"])), decay=decay, freq=freq)


def _retention_prepare(c, seed):
    from umbrella_b200 import ops_seq
    s = _retention_inputs(c, seed)
    s["state"] = torch.zeros(c["seqs"], c["heads"], c["dim"], c["vdim"], device=DEV)
    s["batch"] = ops_seq.RaggedBatch([(i, n, 0, 0) for i, n in enumerate(_lengths(c))], DEV)
    return s


def _retention_run(c, s):
    from umbrella_b200 import ops_seq
    out = ops_seq.retention(s["x"], s["batch"], c["heads"], c["dim"], c["vdim"], c["dim"], s["freq"], s["decay"], _EPS, s["state"],
                            dtype=torch.bfloat16)
    return out, s["state"]


def _retention_exact(c, seed):
    s = _retention_inputs(c, seed)
    H, D, V, at = c["heads"], c["dim"], c["vdim"], 0
    x, lens = s["x"].to(F64), _lengths(c)
    out, state = torch.empty(x.shape[0], H, V, dtype=F64, device=DEV), torch.empty(c["seqs"], H, D, V, dtype=F64, device=DEV)

    def turn(t):
        ang = torch.arange(t.shape[0], dtype=F64, device=DEV)[:, None] * s["freq"].to(F64)[None]
        cs, sn, u, v = torch.cos(ang)[:, None], torch.sin(ang)[:, None], t[..., :D // 2], t[..., D // 2:]
        return torch.cat([u * cs - v * sn, v * cs + u * sn], -1)
    for b, n in enumerate(lens):
        q, k, v, _ = torch.split(x[at:at + n], [H * D, H * D, H * V, H * V], -1)
        q, k, v = turn(q.reshape(n, H, D)), turn(k.reshape(n, H, D)) * D ** -0.5, v.reshape(n, H, V)
        i = torch.arange(n, dtype=F64, device=DEV)
        for h in range(H):
            d = s["decay"][h].to(F64)
            far = (i[:, None] - i[None]).clamp(min=0)
            out[at:at + n, h] = torch.tril((q[:, h] @ k[:, h].T) * d ** far) @ v[:, h]
            state[b, h] = (k[:, h] * (d ** (n - 1 - i))[:, None]).T @ v[:, h]
        at += n
    out = (out / torch.sqrt((out * out).mean(-1, keepdim=True) + _EPS)).reshape(at, H * V)
    gate = x[:, 2 * H * D + H * V:]
    return out * gate * torch.sigmoid(gate), state


def _retention_work(c):
    n, H, D, V = sum(_lengths(c)), c["heads"], c["dim"], c["vdim"]
    return dict(bytes=4 * n * 2 * H * (D + V) + 2 * n * H * V + 4 * c["seqs"] * H * D * V, flops=4 * n * H * D * V)


# ---------------------------------------------------------------------------------------------- INT4 Llama: one layer and the head
_SIZES = {"8b": dict(hidden_size=4096, intermediate_size=14336, num_attention_heads=32, num_key_value_heads=8),
          "70b": dict(hidden_size=8192, intermediate_size=28672, num_attention_heads=64, num_key_value_heads=8)}
_VOCAB, _THETA, _D, _GROUP, _LEPS = 128256, 500000.0, 128, 128, 1e-5


def _llama_dims(c):
    z = _SIZES[c["size"]]
    H, I, kv = z["hidden_size"], z["intermediate_size"], z["num_key_value_heads"] * _D
    return H, I, dict(wq=(H, H), wk=(H, kv), wv=(H, kv), wo=(H, H), gate_proj=(H, I), up_proj=(H, I), down_proj=(I, H))


def _llama_weights(c, seed):
    g, f16 = _gen(seed), torch.float16
    H, _, dims = _llama_dims(c)
    word = lambda *shape: torch.randint(-2 ** 31, 2 ** 31, shape, generator=g, device=DEV).to(torch.int32)
    w = {name: (word(k, n // 8), word(k // _GROUP, n // 8), (0.003 * (0.5 + torch.rand(k // _GROUP, n, generator=g, device=DEV))).to(f16))
         for name, (k, n) in dims.items()}
    for name in ("input_layernorm", "post_attention_layernorm"):
        w[name] = 1 + _randn(g, H, scale=0.1, dtype=f16)
    head = dict(embed=_randn(g, _VOCAB, H, scale=0.02, dtype=f16), head=_randn(g, _VOCAB, H, scale=0.02, dtype=f16),
                norm=1 + _randn(g, H, scale=0.1, dtype=f16))
    return w, head


def _llama_inputs(c, seed):
    g, n = torch.Generator().manual_seed(seed), c["tokens"]
    parent = [-1] + [int(torch.randint(max(0, i - 6), i, (1,), generator=g)) if c["tree"] else i - 1 for i in range(1, n)]
    depth, seen = [0] * n, torch.zeros(n, n, dtype=torch.bool)
    for i in range(n):
        if i:
            depth[i] = depth[parent[i]] + 1
            seen[i] = seen[parent[i]]
        seen[i, i] = True
    ids = torch.randint(0, _VOCAB, (n,), generator=g)
    gd = _gen(seed + 1)
    cap, hk = c["prefix"] + n, _SIZES[c["size"]]["num_key_value_heads"]
    kv = [_randn(gd, cap, hk, _D, dtype=torch.float16) for _ in range(2)]
    return ids.to(DEV), torch.tensor(depth, device=DEV) + c["prefix"], seen, kv


def _llama_prepare(c, seed):
    from umbrella_b200.models import llama
    w, head = _llama_weights(c, seed)
    ids, pos, seen, kv = _llama_inputs(c, seed)
    n = c["tokens"]
    shape = llama.LlamaShape(num_hidden_layers=1, vocab_size=_VOCAB, rope_theta=_THETA, rope_scaling=None, **_SIZES[c["size"]])
    m = llama.LlamaAwq(shape, max_length=c["prefix"] + n, device=DEV)
    m.alloc()
    m.load_head(head["embed"], head["head"], head["norm"])
    m.load_awq_layer(0, w)
    m.k_cache[0].copy_(kv[0].view(m.k_cache[0].shape))
    m.v_cache[0].copy_(kv[1].view(m.v_cache[0].shape))
    words = -(-n // 32)
    bits = torch.zeros(n, words, dtype=torch.int64)
    for j in range(n):
        bits[:, j // 32] |= seen[:, j].to(torch.int64) << (j % 32)
    return dict(model=m, ids=ids, pos=pos, bits=torch.where(bits >= 2 ** 31, bits - 2 ** 32, bits).to(torch.int32).to(DEV))


def _llama_run(c, s):
    m = s["model"]
    m.kv_offset = c["prefix"]
    if c["tree"]:
        logits = m.verify_forward(s["ids"], s["pos"], c["prefix"], s["bits"])
    else:
        logits = m.prefill_forward(s["ids"], s["pos"])
    return logits, m.k_cache, m.v_cache


def _llama_exact(c, seed):
    w, head = _llama_weights(c, seed)
    ids, pos, seen, kv = _llama_inputs(c, seed)
    n, prefix, Hk = c["tokens"], c["prefix"], _SIZES[c["size"]]["num_key_value_heads"]
    order = torch.tensor([0, 4, 1, 5, 2, 6, 3, 7], device=DEV)

    def unpack(t):
        return ((t[:, :, None] >> (4 * order)) & 15).reshape(t.shape[0], -1)

    def lin(x, name):
        q, z, s = w[name]
        out = torch.empty(x.shape[0], s.shape[1], dtype=F64, device=DEV)
        for c0 in range(0, s.shape[1], 4096):
            c1 = min(c0 + 4096, s.shape[1])
            wt = unpack(q[:, c0 // 8:c1 // 8]) - unpack(z[:, c0 // 8:c1 // 8]).repeat_interleave(_GROUP, 0)
            out[:, c0:c1] = x @ (wt.to(F64) * s[:, c0:c1].to(F64).repeat_interleave(_GROUP, 0))
        return out

    def norm(x, weight):
        return x / torch.sqrt((x * x).mean(-1, keepdim=True) + _LEPS) * weight.to(F64)

    ang = pos.to(F64)[:, None] * (_THETA ** (-torch.arange(0, _D, 2, dtype=F64, device=DEV) / _D))[None]
    cs, sn = torch.cos(ang)[:, None], torch.sin(ang)[:, None]

    def turn(t):
        u, v = t[..., :_D // 2], t[..., _D // 2:]
        return torch.cat([u * cs - v * sn, v * cs + u * sn], -1)
    x = head["embed"][ids].to(F64)
    h = norm(x, w["input_layernorm"])
    q, k, v = turn(lin(h, "wq").reshape(n, -1, _D)), turn(lin(h, "wk").reshape(n, Hk, _D)), lin(h, "wv").reshape(n, Hk, _D)
    keys, vals = (torch.cat([old[:prefix].to(F64), new]) for old, new in zip(kv, (k, v)))
    mask = torch.cat([torch.ones(n, prefix, dtype=torch.bool, device=DEV), seen.to(DEV)], 1)
    per = q.shape[1] // Hk
    o = torch.stack([_softmax_rows(q[:, i], keys[:, i // per], vals[:, i // per], mask, _D ** -0.5, None) for i in range(q.shape[1])], 1)
    x = x + lin(o.reshape(n, -1), "wo")
    h = norm(x, w["post_attention_layernorm"])
    x = x + lin(torch.nn.functional.silu(lin(h, "gate_proj")) * lin(h, "up_proj"), "down_proj")
    rows = norm(x if c["tree"] else x[-1:], head["norm"])
    logits = torch.cat([rows @ head["head"][i:i + 16384].to(F64).T for i in range(0, _VOCAB, 16384)], 1)
    return logits, keys[None], vals[None]


def _llama_work(c):
    H, _, dims = _llama_dims(c)
    n, row, out = c["tokens"], _SIZES[c["size"]]["num_key_value_heads"] * _D, c["tokens"] if c["tree"] else 1
    params = sum(k * m for k, m in dims.values())
    seen = c["prefix"] + n / 2
    return dict(bytes=int(params * (0.5 + 2.5 / _GROUP) + 2 * _VOCAB * H + 4 * out * _VOCAB + 4 * row * (c["prefix"] + n) + 2 * n * H),
                flops=int(2 * n * params + 2 * out * _VOCAB * H + 4 * n * seen * H))


# ---------------------------------------------------------------------------------------------- a served batch
def _served_config(c):
    """Matrix-memory layers with a windowed attention layer as every fourth, each with a dense feed-forward."""
    W, heads = c["width"], c["width"] // 128
    mls = dict(type="mlstm", mixer=dict(heads=heads, dim=64, vdim=128, gate_cap=15.0))
    att = dict(type="attention", mixer=dict(heads=heads, kv_heads=max(1, heads // 4), dim=128, vdim=128, scale=128 ** -0.5,
                                            mask=dict(size=1024), rot=dict(dims=64, base=1e6)))
    return dict(architecture="Zedotar", width=W, vocab=8192, norm=dict(eps=1e-6), logit_softcap=30.0,
                layers=[dict(att if i % 4 == 3 else mls, mlp=dict(kind="dense", ff=2 * W)) for i in range(c["layers"])])


def _served_weights(c, seed):
    g, W, bf = _gen(seed), c["width"], torch.bfloat16
    H, G = W // 128, max(1, W // 512)
    r = lambda o, k, gain=1.0: _randn(g, o, k, scale=gain * k ** -0.5, dtype=bf)
    vec = lambda n, mean=0.0, s=0.1: mean + _randn(g, n, scale=s, dtype=bf)
    layers = []
    for i in range(c["layers"]):
        w = dict(norm=vec(W), norm2=vec(W), o=r(W, H * 128, 0.5), dense=(r(2 * W, W), r(2 * W, W), r(W, 2 * W, 0.5)))
        if i % 4 == 3:
            w.update(q=r(H * 128, W), k=r(G * 128, W), v=r(G * 128, W), g=r(H, W), q_b=vec(H * 128), k_b=vec(G * 128), v_b=vec(G * 128))
        else:
            w.update(q=r(H * 64, W), k=r(H * 64, W), v=r(H * 128, W), g=r(H * 128, W), i=r(H, W), f=r(H, W), i_b=vec(H, 0.0, 1.0),
                     f_b=vec(H, 3.0, 1.0), out_norm=vec(H * 128, 1.0))
        layers.append(w)
    return dict(embed=_randn(g, 8192, W, dtype=bf), head=_randn(g, 8192, W, scale=W ** -0.5, dtype=bf), norm=vec(W)), layers


def _served_tokens(c, seed):
    g = torch.Generator().manual_seed(seed)
    return [torch.randint(0, 8192, (n + c["steps"],), generator=g).tolist() for n in _lengths(c)]


def _served_prepare(c, seed):
    from umbrella_b200.models import zedotar
    head, layers = _served_weights(c, seed)
    m = zedotar.Zedotar(zedotar.spec_from_config(_served_config(c)), device=DEV, dtype=torch.bfloat16, slots=c["seqs"],
                        max_tokens=sum(_lengths(c)))
    m.alloc()
    m.load_head(head["embed"], head["head"], head["norm"])
    for i, w in enumerate(layers):
        m.load_layer(i, w)
    return dict(model=m, tokens=_served_tokens(c, seed))


def _served_run(c, s):
    """The prompts in one step, then decode steps that feed each request's next token; logits of every step."""
    m, lens = s["model"], _lengths(c)
    slots = [m.cache.alloc_slot() for _ in lens]
    out = [m.forward([(slot, t[:n], [n - 1]) for slot, t, n in zip(slots, s["tokens"], lens)])]
    for i in range(c["steps"]):
        out.append(m.forward([(slot, [t[n + i]], [0]) for slot, t, n in zip(slots, s["tokens"], lens)]))
    for slot in slots:
        m.cache.free_slot(slot)
    return out


def _served_exact(c, seed):
    head, layers = _served_weights(c, seed)
    lens, toks, W = _lengths(c), _served_tokens(c, seed), c["width"]
    H, G, B, n = W // 128, max(1, W // 512), c["seqs"], max(_lengths(c)) + c["steps"]
    ids = torch.tensor([t + [0] * (n - len(t)) for t in toks], device=DEV)         # causal: what follows a sequence does not matter
    f64 = lambda t: t.to(F64)
    norm = lambda x, w: x / torch.sqrt((x * x).mean(-1, keepdim=True) + 1e-6) * (1 + f64(w))
    unit = lambda x: x / torch.sqrt((x * x).mean(-1, keepdim=True) + 1e-6)
    x = f64(head["embed"][ids])
    ang = torch.arange(n, dtype=F64, device=DEV)[:, None] * (1e6 ** (-torch.arange(0, 64, 2, dtype=F64, device=DEV) / 64))[None]
    cs, sn = torch.cos(ang)[:, None], torch.sin(ang)[:, None]

    def turn(t):
        u, v = t[..., :32], t[..., 32:64]
        return torch.cat([u * cs - v * sn, v * cs + u * sn, t[..., 64:]], -1)

    def mlstm(h, w):
        q, k = (h @ f64(w["q"]).T).reshape(B, n, H, 64) / 8, (h @ f64(w["k"]).T).reshape(B, n, H, 64)
        v = (h @ f64(w["v"]).T).reshape(B, n, H, 128)
        gi = 15 * torch.tanh((h @ f64(w["i"]).T + f64(w["i_b"])) / 15)
        gf = torch.nn.functional.logsigmoid(15 * torch.tanh((h @ f64(w["f"]).T + f64(w["f_b"])) / 15))
        S, m = torch.zeros(B, H, 64, 129, dtype=F64, device=DEV), torch.zeros(B, H, dtype=F64, device=DEV)
        v1, out = torch.cat([v, torch.ones_like(v[..., :1])], -1), []
        for t in range(n):
            new = torch.maximum(gf[:, t] + m, gi[:, t])
            S = torch.exp(gf[:, t] + m - new)[..., None, None] * S + \
                torch.exp(gi[:, t] - new)[..., None, None] * k[:, t, :, :, None] * v1[:, t, :, None]
            m = new
            o = (S * q[:, t, :, :, None]).sum(2)
            out.append(o[..., :128] / (torch.maximum(o[..., 128].abs(), torch.exp(-m)) + 1e-6)[..., None])
        o = unit(torch.stack(out, 1)).reshape(B, n, H * 128)
        return (o * f64(w["out_norm"]) * torch.sigmoid(h @ f64(w["g"]).T)) @ f64(w["o"]).T

    def attention(h, w):
        q, k, v = ((h @ f64(w[a]).T + f64(w[a + "_b"])).reshape(B, n, -1, 128) for a in "qkv")
        q, k = turn(q), turn(k)
        i = torch.arange(n, device=DEV)
        mask = (i[None] <= i[:, None]) & (i[None] > i[:, None] - 1024)
        zero = torch.zeros((), dtype=F64, device=DEV)
        o = torch.stack([torch.stack([_softmax_rows(q[b, :, j], k[b, :, j // (H // G)], v[b, :, j // (H // G)], mask, 128 ** -0.5, zero)
                                      for j in range(H)], 1) for b in range(B)])
        return (o * torch.sigmoid(h @ f64(w["g"]).T)[..., None]).reshape(B, n, H * 128) @ f64(w["o"]).T
    for i, w in enumerate(layers):
        h = norm(x, w["norm"])
        x = x + (attention(h, w) if i % 4 == 3 else mlstm(h, w))
        h, (gate, up, down) = norm(x, w["norm2"]), w["dense"]
        x = x + (torch.nn.functional.gelu(h @ f64(gate).T, approximate="tanh") * (h @ f64(up).T)) @ f64(down).T
    z = norm(x, head["norm"])
    pick = lambda step: torch.stack([z[b, m - 1 + step] for b, m in enumerate(lens)])
    return [30 * torch.tanh(pick(i) @ f64(head["head"]).T / 30) for i in range(c["steps"] + 1)]


def _served_work(c):
    W, n, B = c["width"], sum(_lengths(c)), c["seqs"]
    H, G = W // 128, max(1, W // 512)
    att, mls = c["layers"] // 4, c["layers"] - c["layers"] // 4
    params = c["layers"] * 6 * W * W + att * W * (2 * H * 128 + 2 * G * 128 + H) + mls * W * (2 * H * 64 + 3 * H * 128 + 2 * H)
    steps, tokens = c["steps"] + 1, n + B * c["steps"]
    return dict(bytes=steps * 2 * (params + 8192 * W) + 4 * 8192 * B * steps + 2 * 4 * B * c["steps"] * mls * H * 64 * 129,
                flops=2 * tokens * params + 2 * steps * B * 8192 * W + 4 * tokens * mls * H * 64 * 129)


# ---------------------------------------------------------------------------------------------- by kind
_KINDS = {"linear": (_linear_prepare, _linear_run, _linear_exact, _linear_work),
          "experts": (_experts_prepare, _experts_run, _experts_exact, _experts_work),
          "attention": (_attention_prepare, _attention_run, _attention_exact, _attention_work),
          "latent": (_latent_prepare, _latent_run, _latent_exact, _latent_work),
          "retention": (_retention_prepare, _retention_run, _retention_exact, _retention_work),
          "llama": (_llama_prepare, _llama_run, _llama_exact, _llama_work),
          "served": (_served_prepare, _served_run, _served_exact, _served_work)}


def prepare(case, seed):
    return dict(_KINDS[case["kind"]][0](case, seed), case=case)


def run(state):
    return _KINDS[state["case"]["kind"]][1](state["case"], state)


def exact(case, seed):
    return _KINDS[case["kind"]][2](case, seed)


def work(case):
    return _KINDS[case["kind"]][3](case)


def tolerance(case):
    """About four times what one pass shows against 64 bits: operands and results in the case's 16-bit type, sums in 32 bits."""
    kind = case["kind"]
    if kind == "linear":
        if case["dtype"] == "f32":
            return {"rel": 2.5e-6}
        return {"rel": 1.5e-5 if case["f32_out"] else 7e-3}
    return {"rel": {"experts": 8e-3, "attention": 7e-3, "latent": 7e-3, "retention": 7e-3, "llama": 8e-3, "served": 5e-2}[kind]}
