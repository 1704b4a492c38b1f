"""The tensor-core attention of steps with several tokens per sequence (csrc/seq/seq_attn_tc.cu; bf16 storage) against the
general kernel run in float32 on the same bf16 numbers: every mask, score option and output form, at the sizes where tiles
of 128 rows and 32 keys end.

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
DECODE = [[(0, 1, 0, 0), (1, 1, 31, 0), (2, 1, 32, 0)], [(1, 1, 127, 0)], [(0, 1, 128, 0), (2, 1, 510, 0)], [(2, 1, 700, 0), (0, 1, 33, 0)]]


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
