"""The native way into the library (csrc/seq/calls.cpp) against the wrappers' own: the same bits for every form that it takes, the same
refusals for those it leaves to them."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


class Declines:
    """Stands in for the module and takes no call."""

    def __getattr__(self, name):
        return lambda *a: None


@pytest.fixture
def K():
    from umbrella_b200 import ops_seq
    return ops_seq


def _both(monkeypatch, fn):
    """fn's results by the native way and by the wrapper's, each on inputs of its own (fn makes them)."""
    from umbrella_b200 import _lib_seq as S
    real, taken = S.load_calls(), []

    class Watch:
        def __getattr__(self, name):
            def go(*a):
                out = getattr(real, name)(*a)
                taken.append(out is not None)
                return out
            return go
    out = []
    for calls in (Watch(), Declines()):
        monkeypatch.setattr(S, "calls", calls)
        torch.manual_seed(3)
        r = fn()
        out.append([t for t in (r if isinstance(r, tuple) else (r,)) if t is not None])
    assert taken and all(taken)
    for a, b in zip(*out, strict=True):
        assert a.shape == b.shape and a.dtype == b.dtype and a.stride() == b.stride() and torch.equal(a, b)


def _r(*s, dt=torch.float32):
    return torch.randn(*s, device=DEV).to(dt)


@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("form", ["plain", "f32_out", "strided", "part_of_k", "part_of_n", "dual", "heads", "gaps", "few_of_more", "one_row", "no_rows"])
def test_gemm(monkeypatch, K, dt, form):
    def go():
        a, w = _r(9, 64, dt=dt), _r(48, 64, dt=dt)
        if form == "strided":
            a = _r(9, 96, dt=dt)[:, 16:80]
        kw = dict(f32_out=dict(out_f32=True), part_of_k=dict(k=32), part_of_n=dict(n=40), dual=dict(dual=True, limit=3), few_of_more=dict(rows=7, max_rows=4)).get(form, {})
        if form == "heads":
            return K.gemm(a, _r(4, 24, 16, dt=dt), groups=4, a_goff=16, c_goff=24, n=24, k=16)
        if form == "gaps":
            return K.gemm(a, _r(4, 24, 16, dt=dt), groups=4, a_goff=16, c_goff=32, n=24, k=16, out_f32=True)
        return K.gemm(a[:1] if form == "one_row" else (a[:0] if form == "no_rows" else a), w, **kw)
    _both(monkeypatch, go)


@pytest.mark.parametrize("n,top,width", [(1, 2, 64), (40, 2, 256), (200, 1, 256)])
def test_routed_experts(monkeypatch, K, n, top, width):
    def go():
        from umbrella_b200 import _lib_seq as S
        h, x = _r(n, width, dt=torch.bfloat16), _r(n, width)
        sel_w, off, tok, pos, sel_e = K.moe_route(h, _r(4, width), top)
        order = torch.argsort(tok.long() * 8 + torch.repeat_interleave(torch.arange(4, device=DEV), off.diff().long(), output_size=n * top))     # (within an expert: any order)
        y = K.gemm(h, _r(4, 128, width, dt=torch.bfloat16), groups=4, n=64, dual=True, limit=7.0, grp_off=off, row_src=tok, rows=n * top, max_rows=n)
        o = K.gemm(y, _r(4, width, 64, dt=torch.bfloat16), out_f32=True, groups=4, grp_off=off, rows=n * top, max_rows=n)
        z, copy = K.add_norm(x, _r(width), None, 1e-6, kind=S.UMBS_NORM_RMS, dtype=torch.bfloat16, rows=torch.arange(n, dtype=torch.int32, device=DEV), pair_out=o,
                             sel_w=sel_w, pair_pos=pos, want_copy=True)
        plain = K.add_norm(x, _r(width), _r(width), 1e-5, w_offset=1.0, delta=_r(n, width), scale=_r(width), mult=0.5)
        return sel_w, off, sel_e, y[order], o[order], z, copy, plain, x
    _both(monkeypatch, go)


@pytest.mark.parametrize("tokens,pool,gate", [(1, 0, None), (1, 16, "head"), (40, 16, "column"), (40, 0, "head")])
def test_attention_over_a_cache(monkeypatch, K, tokens, pool, gate):
    def go():
        from umbrella_b200 import _lib_seq as S
        H, G, D, cap = 4, 2, 64, 160
        b = K.RaggedBatch([(0, tokens, 100, 0), (1, tokens, 37, 0)], DEV)
        bf = dict(dt=torch.bfloat16)
        cache, pools = _r(2, cap, 2 * G * D, **bf), _r(2, 10, 2 * G * D, **bf) if pool else None
        g = None if gate is None else _r(2 * tokens, H if gate == "head" else H * D)
        out = K.cached_attention(_r(2 * tokens, H * D, **bf), _r(2 * tokens, 2 * G * D, **bf), cache, b, H, G, D, D, D ** -0.5, mode=S.UMBS_ATTN_SOFTMAX_SINK,
                                 window=64 if pool else 0, pool=pool, pool_cache=pools, gate=g, gate_per_head=gate == "head", sink=_r(H))
        return out, cache, pools
    _both(monkeypatch, go)


@pytest.mark.parametrize("shared,gated", [(0, False), (32, True)])
def test_attention_of_a_step(monkeypatch, K, shared, gated):
    def go():
        b, H, D, n = K.RaggedBatch([(0, 50, 0, 0), (1, 20, 0, 0)], DEV), 4, 64, 70
        bf = dict(dt=torch.bfloat16)
        kv = _r(n, 2 * H * D, **bf)
        return K.window_attention_shared(_r(n, H * (D + shared), **bf), kv[:, :H * D], _r(n, shared, **bf) if shared else None, kv[:, H * D:], b, H, 0.1, window=30,
                                         sink=_r(H) if gated else None, use_sink=gated, gate=_r(n, H * D) if gated else None)
    _both(monkeypatch, go)


@pytest.mark.parametrize("tokens,dt,segments", [(1, torch.bfloat16, True), (200, torch.float32, True), (200, torch.bfloat16, False)])
def test_retention(monkeypatch, K, tokens, dt, segments):
    def go():
        b, H, D, V = K.RaggedBatch([(0, tokens, 0, 0)], DEV), 4, 64, 64
        state = _r(1, H, D, V)
        return K.retention(_r(tokens, 2 * H * (D + V)), b, H, D, V, D, torch.rand(D // 2, device=DEV), torch.full((H,), 0.97, device=DEV), 1e-6, state, dtype=dt,
                           segments=segments), state
    _both(monkeypatch, go)


def test_what_is_not_plain_is_left_to_the_wrapper(K):
    a, w = _r(4, 64, dt=torch.bfloat16), _r(8, 64, dt=torch.bfloat16)
    with pytest.raises(TypeError):
        K.gemm(a.half(), w.half())
    with pytest.raises(AssertionError):
        K.gemm(a, w.float())
    with pytest.raises(AssertionError):
        K.gemm(a, w.T.contiguous().T)
    with pytest.raises(AssertionError):
        K.gemm(a.T.contiguous().T, w)
    with pytest.raises(RuntimeError, match="gemm failed"):
        K.gemm(a, w, limit=1.0, k=-1)

    class Sub(torch.Tensor):
        pass
    assert torch.equal(K.gemm(a.as_subclass(Sub), w), K.gemm(a, w))
