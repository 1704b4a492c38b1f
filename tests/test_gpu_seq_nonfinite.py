"""Infinities and NaNs on the sequence-state decoders' kernels stay where the arithmetic puts them: a token that holds one does
not reach tokens that do not see it, and what plain fp32 arithmetic makes infinite is infinite."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def rnd(*shape, seed=0, scale=1.0):
    return scale * torch.randn(*shape, generator=torch.Generator().manual_seed(seed))


# ---------------------------------------------------------------------------------------------- routing
@pytest.mark.parametrize("mode", ["SOFTMAX_TOP", "SIGMOID_GROUPS", "SOFTMAX_ALL"])
@pytest.mark.parametrize("n,experts", [(5, 16), (16, 16), (70, 16), (1030, 24)])          # one block; four and eight tokens to a block
def test_a_token_without_comparable_scores_leaves_its_neighbours_alone(mode, n, experts):
    from umbrella_b200 import _lib_seq as S, ops_seq as K
    top, width = 3, 64
    h, w = rnd(n, width, seed=1).to(DEV), rnd(experts, width, seed=2).to(DEV)
    bad = sorted({1, n // 2, n - 1})
    route = lambda x: K.moe_route_ex(x, w, top, getattr(S, "UMBS_ROUTE_" + mode), 4, 2)
    want_w, _, _, _, want_e = route(h)
    hn = h.clone()
    hn[bad] = float("nan")
    sel_w, off, tok, pos, sel_e = route(hn)
    good = [i for i in range(n) if i not in bad]
    assert torch.equal(sel_w[good], want_w[good]) and torch.equal(sel_e[good], want_e[good])
    assert torch.isnan(sel_w[bad]).all()
    assert int(sel_e.min()) >= 0 and int(sel_e.max()) < experts
    for i in bad:
        assert len(set(sel_e[i].tolist())) == top                       # an expert of its own for every choice
    assert off.tolist() == [0] + torch.bincount(sel_e.flatten().long(), minlength=experts).cumsum(0).tolist()
    assert sorted(pos.tolist()) == list(range(n * top))
    assert torch.equal(tok[pos.long()].cpu(), torch.arange(n * top).div(top, rounding_mode="floor").int())


# ---------------------------------------------------------------------------------------------- recurrences, 32 tokens at a time
@pytest.mark.parametrize("n", [64, 90, 500])
@pytest.mark.parametrize("kind", ["retention", "mlstm"])
@pytest.mark.parametrize("what", ["row", "values"])
def test_tokens_in_front_of_a_nan_keep_their_bits(kind, n, what):
    from umbrella_b200 import ops_seq as K
    heads, dim, vdim = 2, 64, 128
    hd, hv = heads * dim, heads * vdim
    if kind == "retention":
        x = rnd(n, 2 * (hd + hv), seed=n)
        freq, decay = torch.rand(dim // 2, generator=torch.Generator().manual_seed(0)).to(DEV), torch.tensor([0.97, 0.999], device=DEV)

        def run(t):
            state = torch.zeros(1, heads, dim, vdim, device=DEV)
            return K.retention(t, K.RaggedBatch([(0, n, 0, 0)], DEV), heads, dim, vdim, dim, freq, decay, 1e-6, state)
    else:
        x = rnd(n, 2 * (hd + hv) + 2 * heads, seed=n)
        bias, norm = torch.tensor([0.0, 0.0, 3.0, 1.0], device=DEV), torch.ones(hv, device=DEV)

        def run(t):
            state = torch.zeros(1, heads, dim * (vdim + 1) + 1, device=DEV)
            return K.mlstm(t, bias, K.RaggedBatch([(0, n, 0, 0)], DEV), heads, dim, vdim, 15.0, 1e-6, norm, state)
    x = x.to(DEV)
    want = run(x)
    assert torch.isfinite(want).all()
    for j in (1, 2, 3, 4, 33, 62, n - 1):                            # each place of a group of four rows, both sides of a tile's end
        y = x.clone()
        if what == "row":
            y[j] = float("nan")
        else:
            y[j, 2 * hd:2 * hd + hv] = float("inf")
        out = run(y)
        assert torch.equal(out[:j], want[:j]), j
        assert not torch.isfinite(out[j]).any(), j


@pytest.mark.parametrize("n", [128, 300])
@pytest.mark.parametrize("what", ["state", "row", "values"])
def test_retention_in_pieces_of_128_from_a_carried_state(n, what):
    """What is not finite in a carried state, a row or a token's values is where float64 has it, in the outputs (rows of the norm) and in the state;
    the rest is what it is without.  Tolerance as in test_gpu_seq_chunk.py."""
    from test_gpu_seq_chunk import _ratio, _retention64
    from umbrella_b200 import ops_seq as K
    heads, dim, vdim, j = 2, 64, 128, n // 2
    hd, hv = heads * dim, heads * vdim
    x, state = rnd(n, 2 * (hd + hv), seed=n).to(DEV), rnd(1, heads, dim, vdim, seed=1).to(DEV)
    decay = torch.tensor([0.97, 0.999], device=DEV)

    def run(t, S):
        S = S.clone()
        out = K.retention(t, K.RaggedBatch([(0, n, 5, 0)], DEV), heads, dim, vdim, 0, torch.zeros(1, device=DEV), decay, 1e-6, S, k_scale=1.0)
        return out, S[0]
    clean, clean_state = run(x, state)
    if what == "state":
        state[0, 0, 3, 7] = float("inf")
    elif what == "row":
        x[j, dim:2 * dim] = float("nan")                                # of queries: head 1's row j alone
        x[j, hd + 5] = float("nan")                                     # of keys: head 0 from row j on
    else:
        x[j, 2 * hd + 9] = float("-inf")                                # a value of head 0
    out, got = run(x, state)
    want, S = _retention64(x, heads, dim, vdim, decay, state[0], 1e-6)
    assert torch.equal(torch.isfinite(got), torch.isfinite(S)) and torch.equal(torch.isnan(got), torch.isnan(S))
    fin = torch.isfinite(S)
    assert torch.equal(got[torch.isinf(S)].double(), S[torch.isinf(S)]) and _ratio(got[fin], S[fin]) < 2e-6
    if what == "values":                                                # (a score times an infinity is one; a state's column of them is NaN: a piece later)
        assert not bool(torch.isfinite(out[j:, 9]).any()) and _ratio(out[:, vdim:], want[:, vdim:]) < 2e-6
    else:
        fin = torch.isfinite(want)
        assert torch.equal(torch.isfinite(out), fin) and _ratio(out[fin], want[fin]) < 2e-6
    first = 0 if what == "state" else j
    assert torch.equal(out[:first], clean[:first])
    if what != "row":
        assert torch.equal(out[:, vdim:], clean[:, vdim:]) and torch.equal(got[1], clean_state[1])


# ---------------------------------------------------------------------------------------------- attention
def seen_only(q, keys, values, visible, scale, sink):
    """float64: every row over the keys it sees and no others.  q [n, d], keys [m, d], values [m, e], visible [n, m]."""
    rows = []
    for i in range(q.shape[0]):
        at = visible[i].nonzero().flatten()
        z = (keys[at] @ q[i]) * scale
        m = torch.maximum(z.max(), sink)
        p = torch.exp(z - m)
        rows.append((p[:, None] * values[at]).sum(0) / (p.sum() + torch.exp(sink - m)))
    return torch.stack(rows)


def assert_same(got, want):
    """NaN where it is NaN, infinite where it is infinite, else within the rounding of a bf16 result (2^-8 of the row's largest)."""
    got, want = got.double().cpu(), want.cpu()
    assert torch.equal(torch.isnan(got), torch.isnan(want))
    assert torch.equal(got[torch.isinf(want)], want[torch.isinf(want)]) and torch.equal(torch.isinf(got), torch.isinf(want))
    ok = torch.isfinite(want)
    big = torch.where(ok, want, torch.zeros_like(want)).abs().amax(-1, keepdim=True).expand_as(want)
    assert bool(((got - want).abs()[ok] <= 2.0 ** -8 * big[ok] + 1e-6).all())


BAD = {"value": lambda row, kdim: row[kdim + 3:kdim + 4].fill_(float("inf")),
       "both signs": lambda row, kdim: (row[kdim + 3:kdim + 4].fill_(float("inf")), row[kdim + 5:kdim + 6].fill_(float("-inf"))),
       "token": lambda row, kdim: row.fill_(float("nan"))}


@pytest.mark.parametrize("what", list(BAD))
@pytest.mark.parametrize("tokens,past", [(150, 0), (40, 90), (1, 300), (1, 2000)])           # a prompt, a later portion of one, decode steps
@pytest.mark.parametrize("dim,window", [(64, 0), (72, 50), (128, 100)])
def test_attention_over_a_cache(what, tokens, past, dim, window):
    from umbrella_b200 import _lib_seq as S, ops_seq as K
    heads, kv_heads, n = 4, 2, past + tokens
    kdim = kv_heads * dim
    q = rnd(tokens, heads * dim, seed=1).bfloat16()
    rows = rnd(n, 2 * kdim, seed=2).bfloat16()
    bad = n - 1 if tokens == 1 and window else max(n - 30, past + tokens // 2) if tokens > 1 else n // 2
    for at in sorted({bad, max(bad - 17, 0)}):
        for g in range(kv_heads):
            part = rows[at] if what == "token" else rows[at, kdim + g * dim:kdim + (g + 1) * dim]
            BAD[what](part, 0)
        if what == "token":
            break
    sink = rnd(heads, seed=3)
    cache = torch.zeros(1, max(n, 1), 2 * kdim, dtype=torch.bfloat16)
    cache[0, :past] = rows[:past]
    out = K.cached_attention(q.to(DEV), rows[past:].contiguous().to(DEV), cache.to(DEV), K.RaggedBatch([(0, tokens, past, 0)], DEV), heads, kv_heads,
                             dim, dim, dim ** -0.5, mode=S.UMBS_ATTN_SOFTMAX_SINK, window=window, sink=sink.to(DEV), append=False)
    pos, j = torch.arange(past, n)[:, None], torch.arange(n)[None]
    visible = (j <= pos) & (j > pos - (window or 1 << 30))
    for h in range(heads):
        g = h // (heads // kv_heads)
        want = seen_only(q[:, h * dim:(h + 1) * dim].double(), rows[:, g * dim:(g + 1) * dim].double(), rows[:, kdim + g * dim:kdim + (g + 1) * dim].double(),
                         visible, float(torch.tensor(dim ** -0.5)), sink[h].double())
        assert_same(out[:, h * dim:(h + 1) * dim], want)


@pytest.mark.parametrize("what", list(BAD))
@pytest.mark.parametrize("shared,window", [(0, 0), (64, 40)])
def test_attention_of_a_steps_own_keys(what, shared, window):
    from umbrella_b200 import ops_seq as K
    heads, dim, n = 2, 64, 150
    q, k, v = rnd(n, heads * (dim + shared), seed=1).bfloat16(), rnd(n, heads * dim, seed=2).bfloat16(), rnd(n, heads * dim, seed=3).bfloat16()
    ks = rnd(n, shared, seed=4).bfloat16() if shared else None
    for h in range(heads):
        BAD[what](v[100, h * dim:(h + 1) * dim], 0)
    if what == "token":
        k[100] = float("nan")
    sink = rnd(heads, seed=5)
    out = K.window_attention_shared(q.to(DEV), k.to(DEV), ks.to(DEV) if shared else None, v.to(DEV), K.RaggedBatch([(0, n, 0, 0)], DEV), heads,
                                    (dim + shared) ** -0.5, window=window, sink=sink.to(DEV))
    i = torch.arange(n)
    visible = (i[None] <= i[:, None]) & (i[None] > i[:, None] - (window or 1 << 30))
    for h in range(heads):
        keys = torch.cat([k[:, h * dim:(h + 1) * dim]] + ([ks] if shared else []), 1).double()
        want = seen_only(q[:, h * (dim + shared):(h + 1) * (dim + shared)].double(), keys, v[:, h * dim:(h + 1) * dim].double(), visible,
                         float(torch.tensor((dim + shared) ** -0.5)), sink[h].double())
        assert_same(out[:, h * dim:(h + 1) * dim], want)


@pytest.mark.parametrize("what", list(BAD))
@pytest.mark.parametrize("tokens,past", [(20, 0), (77, 0), (130, 0), (40, 90), (65, 700)])
@pytest.mark.parametrize("dim,window", [(64, 0), (128, 100), (40, 30)])
def test_a_neighbours_numbers_do_not_reach_a_sequence(what, tokens, past, dim, window):
    """Numbers that are not finite in the rows behind a sequence's own leave it as it is, bit for bit: neither in its results nor on the way of the plain
    rows, which sum in another order."""
    from umbrella_b200 import _lib_seq as S, ops_seq as K
    heads, kv_heads, more = 4, 2, 50
    kdim, n = kv_heads * dim, tokens + more
    q, rows = rnd(n, heads * dim, seed=1).bfloat16(), rnd(n, 2 * kdim, seed=2).bfloat16()
    cache = rnd(2, past + tokens + 64, 2 * kdim, seed=4).bfloat16().to(DEV)
    sink = rnd(heads, seed=3).to(DEV)
    bad = rows.clone()
    for at in (tokens, tokens + 3):
        for g in range(kv_heads):
            BAD[what](bad[at] if what == "token" else bad[at, kdim + g * dim:kdim + (g + 1) * dim], 0)
    batch = K.RaggedBatch([(0, tokens, past, 0), (1, more, 0, 0)], DEV)
    cached = [K.cached_attention(q.to(DEV), r.to(DEV), cache, batch, heads, kv_heads, dim, dim, dim ** -0.5, mode=S.UMBS_ATTN_SOFTMAX_SINK, window=window, sink=sink,
                                 append=False)[:tokens] for r in (rows, bad)]
    assert torch.equal(*cached) and bool(torch.isfinite(cached[0]).all())
    if past == 0:
        own = [K.window_attention_shared(q[:, :kdim].contiguous().to(DEV), r[:, :kdim].to(DEV), None, r[:, kdim:].to(DEV), batch, kv_heads, dim ** -0.5, window=window,
                                         use_sink=False)[:tokens] for r in (rows, bad)]
        assert torch.equal(*own)
