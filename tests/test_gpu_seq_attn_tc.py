"""The tensor-core attention of steps with several tokens per sequence (csrc/seq/seq_attn_tc.cu; bf16 storage) against the
general kernel run in float32 on the same bf16 numbers: every mask, score option and output form, at the sizes where tiles
of 128 rows and 64 keys end.

Tolerance: both sum exact products of bf16 numbers in fp32; what is left is the rounding of the bf16 result, at most 2^-8 of a
value and so of the norm (the weights' and sums' 32-bit errors are below 1e-4 of that)."""
import ctypes

import pytest
import torch

import seq_helpers as H

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
TOL = 2.0 ** -8


def _r(g, *shape, s=1.0):
    return (torch.randn(*shape, generator=g, device=DEV) * s).bfloat16()


@pytest.fixture(scope="module")
def ops():
    from umbrella_b200 import _lib_seq, ops_seq
    yield ops_seq
    assert _lib_seq.load().umbs_kernel_timeouts() == 0


# (slot, tokens, position of the first): fresh, later portions, more than a tile, one row among them, a ring that wraps
STEPS = {"fresh": [(2, 128, 0, 0), (0, 65, 0, 0), (1, 1, 0, 0)], "long": [(1, 300, 0, 0)],
         "portion": [(0, 129, 63, 0), (2, 7, 200, 0)], "one": [(0, 2, 64, 0)]}


def _scored(ops, q, kv, cache, batch, heads, kv_heads, dim, vdim, scale, window=0, softcap=0.0, r1=None, r2=None, chunk=0, gate=None):
    """Score options with the result in q's type (fp32 results for a finishing pass stay with the fp32 kernels)."""
    from umbrella_b200 import _lib_seq as S
    out, p = torch.empty(q.shape[0], heads * vdim, dtype=q.dtype, device=q.device), ops._p
    part = torch.empty(2048 * (vdim + 2), device=q.device)
    o = S.AttnOpts()
    o.softcap, o.chunk, o.maps, o.value_heads = softcap, chunk, 1, 1
    o.dist_r1, o.dist_r2 = (r.data_ptr() if r is not None else None for r in (r1, r2))
    S.check(S.load().umbs_cached_attention_ex(ops._mode(q), S.UMBS_ATTN_SOFTMAX, p(q), p(kv), p(cache), cache.shape[1], None, 0, ctypes.byref(batch.c),
                                              heads, kv_heads, dim, vdim, window, 0, float(scale), None, p(gate),
                                              gate.stride(0) if gate is not None else 0, 0, ctypes.byref(o), p(part), part.numel() * 4, p(out),
                                              ops._stream()), "cached_attention_ex")
    return out


def _cached(ops, dt, seqs, heads, kv_heads, dim, vdim, seed=3, ring=512, pool=0, opts=(), **kw):
    g = torch.Generator(device=DEV).manual_seed(seed)
    T, row = sum(s[1] for s in seqs), kv_heads * (dim + vdim)
    q = _r(g, T, heads * dim, s=1.5).to(dt)
    kv, cache = _r(g, T, row).to(dt), _r(g, 3, ring, row).to(dt)
    gate = torch.randn(T, heads * vdim + 2, generator=g, device=DEV)
    head = torch.randn(heads, generator=g, device=DEV)
    batch = ops.RaggedBatch(seqs, DEV)
    if pool:
        kw.update(pool=pool, pool_cache=_r(g, 3, 704 // pool + 1, row).to(dt))       # every position of the steps below
    if "sink" in opts:
        kw["sink"] = head
    if "bias" in opts:
        kw["head_bias"] = head
    if "gate" in opts:
        kw["gate"] = gate[:, :heads * vdim] if "unaligned" in opts else gate[:, :heads * vdim].contiguous()
    if "gate_head" in opts:
        kw.update(gate=gate[:, :heads], gate_per_head=True)
    if "dist" in opts:
        kw.update(r1=head.abs(), r2=head.abs() * 0.1)
    fn = (lambda *a, **k: _scored(ops, *a, **k)) if "scored" in opts else ops.cached_attention
    return fn(q, kv, cache, batch, heads, kv_heads, dim, vdim, dim ** -0.5, **kw)


def _both(ops, *a, **kw):
    got, ref = _cached(ops, torch.bfloat16, *a, **kw), _cached(ops, torch.float32, *a, **kw)
    assert torch.isfinite(got.float()).all()
    assert H.rel_err(got, ref.cpu()) < TOL


@pytest.mark.parametrize("step", STEPS)
@pytest.mark.parametrize("dim,vdim", [(128, 128), (64, 64), (8, 8), (72, 96), (192, 40)])
def test_sizes(ops, step, dim, vdim):
    _both(ops, STEPS[step], 4, 2, dim, vdim)


@pytest.mark.parametrize("window", [1, 63, 64, 65, 128, 200])
def test_windows(ops, window):
    for step in STEPS.values():
        _both(ops, step, 2, 1, 64, 64, window=window)


@pytest.mark.parametrize("window,pool", [(1, 4), (33, 16), (64, 64)])
def test_pooled_blocks_and_sinks(ops, window, pool):
    from umbrella_b200 import _lib_seq as S
    for step in STEPS.values():
        _both(ops, step, 4, 4, 64, 128, window=window, pool=pool, mode=S.UMBS_ATTN_SOFTMAX_SINK, opts=("sink", "gate_head"))


def test_sigmoid_weights(ops):
    from umbrella_b200 import _lib_seq as S
    for step in STEPS.values():
        for window in (0, 70):
            _both(ops, step, 4, 2, 64, 64, window=window, mode=S.UMBS_ATTN_SIGMOID, opts=("bias", "gate"))
    _both(ops, STEPS["fresh"], 4, 2, 64, 64, opts=("gate", "unaligned"))


@pytest.mark.parametrize("kw,opts", [(dict(softcap=5.0), ()), (dict(), ("dist",)), (dict(chunk=48), ("gate",)), (dict(chunk=128, window=100), ()),
                                     (dict(softcap=20.0), ("dist", "gate"))])
def test_score_options(ops, kw, opts):
    for step in STEPS.values():
        _both(ops, step, 4, 2, 64, 32, opts=opts + ("scored",), **kw)


def test_a_ring_that_wraps(ops):
    _both(ops, [(1, 40, 130, 0), (0, 130, 61, 0)], 4, 2, 64, 64, window=64, ring=104)


def test_the_reference_moves_late_and_far(ops):
    """Scores that grow along the keys by far more than the reference may lag behind, and a first tile that is hidden to most rows."""
    T, D = 400, 64
    g = torch.Generator(device=DEV).manual_seed(5)
    for dt in (torch.bfloat16, torch.float32):
        k = torch.ones(T, D, device=DEV) * torch.linspace(-20, 40, T, device=DEV)[:, None] / 8
        kv = torch.cat([k, torch.randn(T, D, generator=g.manual_seed(6), device=DEV)], 1).bfloat16().to(dt)
        out = ops.cached_attention(torch.ones(T, D, device=DEV, dtype=dt), kv, torch.zeros(1, 512, 2 * D, device=DEV, dtype=dt),
                                   ops.RaggedBatch([(0, T, 0, 0)], DEV), 1, 1, D, D, 1.0, window=130)
        if dt == torch.bfloat16:
            got = out
    assert H.rel_err(got, out.cpu()) < TOL


@pytest.mark.parametrize("dim,shared,vdim", [(128, 64, 128), (64, 0, 128), (64, 32, 64), (8, 8, 8), (120, 72, 104)])
def test_keys_of_the_step(ops, dim, shared, vdim):
    Hh = 3
    seqs = [(0, 200, 0, 0), (1, 1, 0, 0), (2, 129, 0, 0)]
    T = 330
    g = torch.Generator(device=DEV).manual_seed(7)
    q, kv, ks = _r(g, T, Hh * (dim + shared)), _r(g, T, Hh * (dim + vdim)), _r(g, T, shared) if shared else None
    sink, gate = torch.randn(Hh, generator=g, device=DEV), torch.randn(T, Hh * vdim, generator=g, device=DEV)
    batch = ops.RaggedBatch(seqs, DEV)
    for kw in (dict(use_sink=False), dict(sink=sink, gate=gate), dict(window=65, gate=gate[:, :Hh], gate_per_head=True)):
        got, ref = (ops.window_attention_shared(q.to(dt), kv[:, :Hh * dim].to(dt), ks.to(dt) if shared else None, kv[:, Hh * dim:].to(dt), batch,
                                                Hh, (dim + shared) ** -0.5, **kw) for dt in (torch.bfloat16, torch.float32))
        assert H.rel_err(got, ref.cpu()) < TOL


# ---------------------------------------------------------------------------------------------- decode steps
# one token per sequence: the first token, a tile of 32 keys and its edges, several tiles per warp, splits, a ring that wraps
DECODE = [[(0, 1, 0, 0), (1, 1, 31, 0), (2, 1, 32, 0)], [(1, 1, 127, 0)], [(0, 1, 128, 0), (2, 1, 510, 0)], [(2, 1, 700, 0), (0, 1, 33, 0)],
          [(0, 1, 0, 0), (1, 1, 31, 0), (2, 1, 200, 0)]]


@pytest.mark.parametrize("heads,kv_heads", [(1, 1), (4, 2), (6, 2), (16, 2), (10, 2)])
@pytest.mark.parametrize("dim,vdim", [(128, 128), (64, 40), (8, 8), (104, 72)])
def test_decode_sizes(ops, heads, kv_heads, dim, vdim):
    for step in DECODE:
        _both(ops, step, heads, kv_heads, dim, vdim, window=0 if step[0][2] < 600 else 500)


@pytest.mark.parametrize("window,pool", [(1, 4), (33, 16), (300, 0)])
def test_decode_masks_and_outputs(ops, window, pool):
    from umbrella_b200 import _lib_seq as S
    for step in DECODE:
        _both(ops, step, 8, 2, 64, 64, window=window, pool=pool, mode=S.UMBS_ATTN_SOFTMAX_SINK, opts=("sink", "gate_head"))
        _both(ops, step, 8, 2, 64, 64, window=window, pool=pool, mode=S.UMBS_ATTN_SIGMOID, opts=("bias", "gate"))
        _both(ops, step, 8, 2, 64, 64, window=window, pool=pool, mode=S.UMBS_ATTN_SOFTMAX_SINK, opts=("sink",), split=False)


@pytest.mark.parametrize("kw,opts", [(dict(softcap=5.0), ("dist",)), (dict(chunk=48), ("gate",))])
def test_decode_score_options(ops, kw, opts):
    for step in DECODE[:3]:
        _both(ops, step, 4, 2, 64, 32, opts=opts + ("scored",), **kw)


@pytest.mark.parametrize("which", ["k", "v", "ks", "same"])
def test_overlapping_rows_of_a_steps_keys_are_taken(ops, which):
    """Rows that share memory (each a few numbers behind the one before it, or one row for every token) give what copies of them give."""
    heads, dim, shared, vdim, T = 2, 64, 64, 64, 150
    g = torch.Generator(device=DEV).manual_seed(5)
    rows = dict(q=_r(g, T, heads * (dim + shared), s=1.5), k=_r(g, T, heads * dim), ks=_r(g, T, shared), v=_r(g, T, heads * vdim))
    for name in ("k", "v") if which == "same" else (which,):
        n = rows[name].shape[1]
        rows[name] = rows[name][:1].expand(T, n) if which == "same" else _r(g, 8 * T + n).as_strided((T, n), (8, 1))
    batch = ops.RaggedBatch([(0, T - 20, 0, 0), (1, 20, 0, 0)], DEV)
    run = lambda q, k, ks, v: ops.window_attention_shared(q, k, ks, v, batch, heads, (dim + shared) ** -0.5)
    assert torch.equal(run(**rows), run(**{n: t.contiguous() for n, t in rows.items()}))


# ---------------------------------------------------------------------------------------------- against a plain statement in 64 bits
def _plain64(q, rows, pools, pos0, kv_heads, dim, vdim, heads, window=0, pool=0, mode="softmax", sink=None, bias=None, softcap=0.0, r1=None, r2=None, chunk=0):
    """One sequence: q [n, heads dim], rows [pos0 + n, kv_heads (dim + vdim)] of positions 0 .., pools [blocks, same].  Everything double."""
    n, scale, out = q.shape[0], float(torch.tensor(dim ** -0.5)), []
    pos, j = pos0 + torch.arange(n)[:, None], torch.arange(pos0 + n)[None]
    see = (j <= pos) & (j > pos - (window or 1 << 30))
    if chunk:
        see &= j // chunk == pos // chunk
    dist, keys = (pos - j).clamp(min=0), rows
    if pool:
        keys = torch.cat([rows, pools])
        see = torch.cat([see, (torch.arange(pools.shape[0])[None] + 1) * pool <= pos - window + 1], 1)
        dist = torch.cat([dist, torch.zeros(n, pools.shape[0], dtype=torch.long)], 1)
    for h in range(heads):
        g = h // (heads // kv_heads)
        k, v = keys[:, g * dim:(g + 1) * dim], keys[:, kv_heads * dim + g * vdim:kv_heads * dim + (g + 1) * vdim]
        z = q[:, h * dim:(h + 1) * dim] @ k.T * scale
        if mode == "sigmoid":
            out.append((torch.sigmoid(z + bias[h]) * see) @ v)
            continue
        if softcap:
            z = softcap * torch.tanh(z / softcap)
        if r1 is not None:
            z = z - r1[h] * torch.log1p(r2[h] * dist)
        z = z.masked_fill(~see, -float("inf"))
        z = torch.cat([z, sink[h].expand(n, 1)], 1) if sink is not None else z
        out.append(torch.softmax(z, 1)[:, :keys.shape[0]] @ v)
    return torch.cat(out, 1)


@pytest.mark.parametrize("seqs", [[(0, 140, 70, 0), (2, 3, 0, 0)], [(1, 300, 0, 0)], [(0, 1, 200, 0), (1, 1, 5, 0)]])
@pytest.mark.parametrize("dim,vdim", [(128, 128), (72, 40)])
@pytest.mark.parametrize("kw", [dict(), dict(window=50, pool=16, sink=True), dict(window=70, mode="sigmoid"), dict(softcap=5.0, dist=True), dict(chunk=48)],
                         ids=lambda k: "-".join(k) or "plain")
def test_against_float64(ops, seqs, dim, vdim, kw):
    from umbrella_b200 import _lib_seq as S
    kw, heads, kv_heads, ring = dict(kw), 4, 2, 320
    g = torch.Generator(device=DEV).manual_seed(dim)
    T, row = sum(s[1] for s in seqs), kv_heads * (dim + vdim)
    q, kv, cache = _r(g, T, heads * dim, s=1.5), _r(g, T, row), _r(g, 3, ring, row)
    head = torch.randn(heads, generator=g, device=DEV)
    plain = {k: v for k, v in kw.items() if k in ("window", "pool", "mode", "softcap", "chunk")}
    before, batch, pools = cache.clone(), ops.RaggedBatch(seqs, DEV), None
    if kw.get("pool"):
        p = kw["pool"]
        pools = cache.reshape(3, ring // p, p, row).float().mean(2).bfloat16()             # what earlier steps left
    if kw.get("softcap") or kw.get("chunk"):
        r = dict(r1=head.abs(), r2=head.abs() * 0.1) if kw.pop("dist", False) else {}
        plain.update({n: t.double().cpu() for n, t in r.items()})
        got = _scored(ops, q, kv, cache, batch, heads, kv_heads, dim, vdim, dim ** -0.5, **kw, **r)
    else:
        extra = dict(sink=head) if kw.pop("sink", False) else dict(head_bias=head) if kw.get("mode") else {}
        plain.update({"sink" if "sink" in extra else "bias": head.double().cpu()} if extra else {})
        mode = {"sigmoid": S.UMBS_ATTN_SIGMOID, None: S.UMBS_ATTN_SOFTMAX_SINK if "sink" in extra else S.UMBS_ATTN_SOFTMAX}[kw.pop("mode", None)]
        got = ops.cached_attention(q, kv, cache, batch, heads, kv_heads, dim, vdim, dim ** -0.5, mode=mode, pool_cache=pools, append=False, **extra, **kw)
    at = 0
    for slot, n, pos0, _ in seqs:
        rows = torch.cat([before[slot, :pos0], kv[at:at + n]]).double().cpu()
        blocks = (pos0 + n) // kw["pool"] if kw.get("pool") else 0
        ref = _plain64(q[at:at + n].double().cpu(), rows, pools[slot, :blocks].double().cpu() if blocks else rows[:0], pos0, kv_heads, dim, vdim, heads, **plain)
        assert H.rel_err(got[at:at + n], ref) < TOL
        at += n


def test_decode_split_is_one_that_the_scratch_holds(ops):
    """64 sequences of 1055 keys, 16 heads over 4: three splits cost less than one and two cost more (rounds of blocks on the chip), so
    with room for two the step is not split (one launch), with room for three it is (the second launch merges)."""
    from umbrella_b200 import _lib_seq as S
    n, heads, kv_heads, dim = 64, 16, 4, 64
    g = torch.Generator(device=DEV).manual_seed(9)
    q, kv, cache = _r(g, n, heads * dim), _r(g, n, 2 * kv_heads * dim), _r(g, n, 1055, 2 * kv_heads * dim)
    batch, p, lib, outs = ops.RaggedBatch([(i, 1, 1054, 0) for i in range(n)], DEV), ops._p, S.load(), []
    part = torch.empty(3 * n * heads * (dim + 2), device=DEV)
    for room, launches in ((0, 1), (1, 1), (2, 1), (3, 2)):
        out, before = torch.empty(n, heads * dim, dtype=torch.bfloat16, device=DEV), lib.umbs_launch_count()
        S.check(lib.umbs_cached_attention(S.UMBS_BF16, S.UMBS_ATTN_SOFTMAX, p(q), p(kv), p(cache), 1055, None, 0, ctypes.byref(batch.c), heads, kv_heads, dim, dim,
                                          0, 0, dim ** -0.5, None, None, 0, 0, p(part) if room else None, 4 * room * n * heads * (dim + 2), p(out), ops._stream()))
        assert lib.umbs_launch_count() - before == launches, room
        outs.append(out)
    for out in outs[1:]:
        assert H.rel_err(out, outs[0].cpu()) < TOL


@pytest.mark.parametrize("heads,kv_heads,dim", [(16, 4, 128), (16, 4, 64), (8, 8, 64)])
@pytest.mark.parametrize("keys", [1, 16, 17, 32, 33, 64, 65])
def test_decode_steps_of_few_keys(ops, heads, kv_heads, dim, keys):
    """Both kernels on either side of the line between them, and a step captured with few keys whose graph is replayed with many."""
    for n in (1, 3):
        _both(ops, [(i, 1, keys - 1 - i if keys > i else 0, 0) for i in range(n)], heads, kv_heads, dim, dim)
    g = torch.Generator(device=DEV).manual_seed(11)
    q, kv, cache = _r(g, 2, heads * dim, s=1.5), _r(g, 2, 2 * kv_heads * dim), _r(g, 2, 512, 2 * kv_heads * dim)
    short, far = ops.RaggedBatch([(0, 1, keys - 1, 0), (1, 1, 0, 0)], DEV), ops.RaggedBatch([(0, 1, 300, 0), (1, 1, 511, 0)], DEV)
    run = lambda b: ops.cached_attention(q, kv, cache, b, heads, kv_heads, dim, dim, dim ** -0.5, append=False)
    want = [run(short), run(far)]
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = run(short)
    for b, ref in zip((short, far), want):
        for name, t in b.t.items():
            short.t[name].copy_(t)
        graph.replay()
        assert H.rel_err(out, ref.cpu()) < TOL


# (tokens, position of the first): whole tiles of 64 keys and one key less and more, of the step, of the ring and of both; more rows than a block
ENDS = [(63, 0), (64, 0), (127, 0), (129, 0), (191, 0), (193, 0), (2, 62), (2, 63), (2, 126), (40, 64), (64, 128), (65, 127), (129, 191)]


@pytest.mark.parametrize("dim,vdim", [(40, 64), (64, 128), (128, 128), (192, 128)])         # two places for keys and values; one for keys; one for either
@pytest.mark.parametrize("window", [0, 64, 100])
def test_ends_of_key_tiles(ops, dim, vdim, window):
    """Tiles that come by tensor map, the one between ring and step that is copied row by row, and both in turn with one place for them."""
    for tokens, past in ENDS:
        _both(ops, [(1, tokens, past, 0), (0, 3, past // 2, 0)], 4, 2, dim, vdim, window=window)
        if window:
            _both(ops, [(1, tokens, past, 0)], 2, 2, dim, vdim, window=window, pool=16)


@pytest.mark.parametrize("slots,ring", [(1, 128), (3, 192), (2, 100)])
def test_a_cache_that_ends_with_its_allocation(ops, slots, ring):
    """The ring's tensor map ends with the memory that the cache is in: its last slot's last rows are read, and nothing behind them."""
    heads, dim = 2, 64
    g = torch.Generator(device=DEV).manual_seed(3)
    T, row = 70, 2 * heads * dim
    q, kv = _r(g, T, heads * dim), _r(g, T, row)
    cache = _r(g, slots, ring, row)
    assert cache.untyped_storage().nbytes() == cache.numel() * 2
    batch = ops.RaggedBatch([(slots - 1, T, ring, 0)], DEV)
    out = [ops.cached_attention(q.to(dt), kv.to(dt), cache.to(dt), batch, heads, heads, dim, dim, dim ** -0.5, window=ring, append=False) for dt in (torch.bfloat16, torch.float32)]
    assert torch.isfinite(out[0].float()).all() and H.rel_err(out[0], out[1].cpu()) < TOL


@pytest.mark.parametrize("own_keys", [False, True])
def test_gates_are_rounded_quotients(ops, own_keys):
    """A row that sees itself alone with a score of 0 is its value times its gates: fp32 1 / (1 + e^-g) rounded once, bit for bit, down to the quotients
    below the smallest normal number (where an approximate reciprocal is 0)."""
    T, heads, D = 2048, 16, 128
    batch = ops.RaggedBatch([(0, T, 0, 0)], DEV)
    g = torch.Generator(device=DEV).manual_seed(5)
    q, k, v = torch.zeros(T, heads * D, device=DEV).bfloat16(), _r(g, T, heads * D), _r(g, T, heads * D, s=1e4)
    gate = torch.randn(T, heads * D, generator=g, device=DEV) * 2
    gate[:, ::16] = -87 - 1.7 * torch.rand(T, heads * D // 16, generator=g, device=DEV)
    if own_keys:
        got = ops.window_attention_shared(q, k, None, v, batch, heads, 1.0, window=1, use_sink=False, gate=gate)
    else:
        got = ops.cached_attention(q, torch.cat([k, v], 1), torch.zeros(1, 8, 2 * heads * D, device=DEV).bfloat16(), batch, heads, heads, D, D, 1.0, window=1,
                                   gate=gate, append=False)
    assert torch.equal(got, (v.float() * (1 / (1 + torch.exp(-gate)))).bfloat16())
