"""Recurrences taken 32 tokens at a time (csrc/seq/seq_chunk.cu; steps whose longest sequence has 64 tokens or more) against
the walk token by token: the same sequences fed in steps of fewer than 64 tokens.

Tolerance: both add the same fp32 products in another order, over sums that the decays keep to some hundreds of terms; random
signs give about sqrt(500) 2^-24 = 1.3e-6 of a row's norm, 1e-5 leaves room for rows that nearly cancel."""
import pytest
import torch

import seq_helpers as H

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
LENS = [(64,), (65, 1), (95, 200, 31), (500,), (129, 128, 127)]


def _feed(fn, lens, size, x):
    """The sequences' tokens (rows of x, one sequence after the other) in steps of at most `size` per sequence; -> rows in x's order."""
    from umbrella_b200 import ops_seq as K
    starts = [sum(lens[:i]) for i in range(len(lens))]
    out, at = [None] * len(lens), [0] * len(lens)
    while any(a < n for a, n in zip(at, lens)):
        desc, rows = [], []
        for s, n in enumerate(lens):
            m = min(size, n - at[s])
            if m:
                desc.append((s, m, at[s], 0))
                rows.append(torch.arange(starts[s] + at[s], starts[s] + at[s] + m))
        idx = torch.cat(rows)
        y, o = fn(x[idx.to(DEV)].contiguous(), K.RaggedBatch(desc, DEV)), 0
        for s, m, _, _ in desc:
            out[s] = y[o:o + m] if out[s] is None else torch.cat([out[s], y[o:o + m]])
            o += m
            at[s] += m
    return torch.cat(out)


@pytest.mark.parametrize("lens", LENS)
@pytest.mark.parametrize("dim,vdim,rot", [(64, 128, 64), (32, 64, 12), (24, 64, 12), (36, 64, 0), (4, 4, 0), (60, 132, 60)])
def test_retention(lens, dim, vdim, rot):
    from umbrella_b200 import ops_seq as K
    heads = 3
    g = torch.Generator().manual_seed(sum(lens) + dim)
    x = torch.randn(sum(lens), 2 * heads * (dim + vdim), generator=g).to(DEV)
    decay = torch.tensor([0.97, 0.999, 0.5], device=DEV)
    freq = (1e4 ** (-torch.arange(0, max(rot, 2), 2) / max(rot, 2))).float().to(DEV)
    got = []
    for size in (40, 10 ** 6, 70):
        state = torch.full((len(lens), heads, dim, vdim), 3.0, device=DEV)           # dirty: a fresh sequence must not read it
        y = _feed(lambda r, b: K.retention(r, b, heads, dim, vdim, rot, freq, decay, 1e-6, state), lens, size, x)
        got.append((y, state.clone()))
    for y, state in got[1:]:
        assert H.rel_err(y, got[0][0]) < 1e-5 and H.rel_err(state, got[0][1]) < 1e-5


# pieces of 128 tokens (csrc/seq/seq_chunk_tc.cu): key and value sizes in eights and rotations in sixteens; a piece's edges, values in
# one block of 128 columns and in two, a norm per head (in the kernel where a head is one block) and over all heads
@pytest.mark.parametrize("lens", [(128,), (300, 1, 128), (255, 257, 383)])
@pytest.mark.parametrize("dim,vdim,rot", [(8, 8, 0), (64, 72, 48), (40, 136, 32), (64, 128, 64)])
@pytest.mark.parametrize("all_heads", [False, True])
def test_retention_in_pieces_of_128(lens, dim, vdim, rot, all_heads):
    from umbrella_b200 import ops_seq as K
    heads = 3
    g = torch.Generator().manual_seed(sum(lens) + dim)
    x = torch.randn(sum(lens), 2 * heads * (dim + vdim), generator=g).to(DEV)
    decay = torch.tensor([0.97, 0.9995, 0.1], device=DEV)
    freq = (1e4 ** (-torch.arange(0, max(rot, 2), 2) / max(rot, 2))).float().to(DEV)
    w = (1 + 0.1 * torch.randn(heads * vdim, generator=g)).to(DEV) if all_heads else None
    got = []
    for size in (40, 10 ** 6, 150):
        state = torch.full((len(lens), heads, dim, vdim), 3.0, device=DEV)
        y = _feed(lambda r, b: K.retention(r, b, heads, dim, vdim, rot, freq, decay, 1e-6, state, norm_w=w), lens, size, x)
        got.append((y, state.clone()))
    for y, state in got[1:]:
        assert H.rel_err(y, got[0][0]) < 1e-5 and H.rel_err(state, got[0][1]) < 1e-5
    bf = K.retention(x, K.RaggedBatch([(i, n, 0, 0) for i, n in enumerate(lens)], DEV), heads, dim, vdim, rot, freq, decay, 1e-6, state,
                     dtype=torch.bfloat16, norm_w=w)
    assert H.rel_err(bf, got[0][0]) < 2.0 ** -8


@pytest.mark.parametrize("lens", LENS)
@pytest.mark.parametrize("dim,vdim", [(64, 128), (32, 64), (24, 64), (36, 64), (4, 4), (60, 132)])
def test_mlstm(lens, dim, vdim):
    from umbrella_b200 import ops_seq as K
    heads = 2
    g = torch.Generator().manual_seed(sum(lens) + dim)
    x = torch.randn(sum(lens), 2 * heads * dim + 2 * heads * vdim + 2 * heads, generator=g)
    x[:, -2 * heads:] *= 4                                # gates that open and shut
    x, bias = x.to(DEV), torch.tensor([0.0, -2.0, 3.0, 1.0], device=DEV)
    norm = torch.ones(heads * vdim, device=DEV)
    got = []
    for size in (40, 10 ** 6, 70):
        state = torch.full((len(lens), heads, dim * (vdim + 1) + 1), 3.0, device=DEV)
        y = _feed(lambda r, b: K.mlstm(r, bias, b, heads, dim, vdim, 15.0, 1e-6, norm, state), lens, size, x)
        got.append((y, state.clone()))
    for y, state in got[1:]:
        assert H.rel_err(y, got[0][0]) < 1e-5 and H.rel_err(state, got[0][1]) < 1e-5


@pytest.mark.parametrize("vdim", [1, 32, 33, 64, 65, 128, 129, 255, 256, 257, 600])
def test_mlstm_rows_around_a_lanes_columns(vdim):
    """The last kernel takes 32, 64, 128 or 256 columns at a time.  Tolerance: fp32 sums of a few dozen terms and one division, as in the
    operator's own tests."""
    from test_gpu_zed_ops import f32, mlstm_reference, rnd
    from umbrella_b200 import ops_seq as K
    heads, dim, n = 2, 16, 3
    proj, bias, norm = rnd(n, 2 * heads * (dim + vdim + 1), seed=60), rnd(2 * heads, seed=61), 1.0 + rnd(heads * vdim, seed=62, scale=0.2)
    state = torch.zeros(1, heads, dim * (vdim + 1) + 1, device=DEV)
    out = K.mlstm(f32(proj), f32(bias), K.RaggedBatch([(0, n, 0, 0)], DEV), heads, dim, vdim, 10.0, 1e-5, f32(norm), state)
    ref = mlstm_reference(proj, bias, heads, dim, vdim, 10.0, 1e-5, norm)
    assert float((out.double().cpu() - ref.double()).abs().max() / ref.double().abs().max()) < 2e-5


# ---------------------------------------------------------------------------------------------- against the plain recurrences in 64 bits
# (tolerances as in the operators' own tests of shorter steps, test_gpu_seq_ops.py and test_gpu_zed_ops.py)
@pytest.mark.parametrize("dim,vdim,rot,n", [(64, 128, 64, 200), (60, 132, 12, 64), (4, 4, 0, 97)])
def test_retention_against_float64(dim, vdim, rot, n):
    from test_gpu_seq_ops import _ret_inputs, _ret_ref
    from umbrella_b200 import ops_seq as K
    from umbrella_b200.models.seq_model import rotary_inv_freq
    heads, decay, base = 2, [0.93, 0.9995], 50.0
    qkvg, q, k, v, gate = _ret_inputs(n, heads, dim, vdim, 21)
    state = torch.full((1, heads, dim, vdim), 5.0, device=DEV)
    out = K.retention(qkvg.to(DEV), K.RaggedBatch([(0, n, 0, 0)], DEV), heads, dim, vdim, rot, (rotary_inv_freq(rot, base) if rot else torch.zeros(1)).to(DEV),
                      torch.tensor(decay, device=DEV), 1e-4, state)
    assert H.row_err(out, _ret_ref(q, k, v, gate, dim, rot, base, decay, 1e-4)) < 2e-5


@pytest.mark.parametrize("dim,vdim,n", [(64, 128, 200), (60, 132, 64), (4, 4, 97)])
def test_mlstm_against_float64(dim, vdim, n):
    from test_gpu_zed_ops import f32, mlstm_reference, rnd
    from umbrella_b200 import ops_seq as K
    heads = 2
    proj, bias, norm = rnd(n, 2 * heads * (dim + vdim + 1), seed=70), rnd(2 * heads, seed=71), 1.0 + rnd(heads * vdim, seed=72, scale=0.2)
    state = torch.full((1, heads, dim * (vdim + 1) + 1), 2.5, device=DEV)
    out = K.mlstm(f32(proj), f32(bias), K.RaggedBatch([(0, n, 0, 0)], DEV), heads, dim, vdim, 10.0, 1e-5, f32(norm), state)
    ref = mlstm_reference(proj, bias, heads, dim, vdim, 10.0, 1e-5, norm)
    assert float((out.double().cpu() - ref.double()).abs().max() / ref.double().abs().max()) < 2e-5


def _retention64(x, heads, dim, vdim, decay, S, eps):
    """float64, token by token, no rotation, keys as they are; -> gated rows of unit norm, the state behind them"""
    n, hd, hv = x.shape[0], heads * dim, heads * vdim
    q, k, v, gate = x.double().split([hd, hd, hv, hv], 1)
    q, k, v = q.view(n, heads, dim), k.view(n, heads, dim), v.view(n, heads, vdim)
    S, out, d = S.double(), [], decay.double()[:, None, None]
    for t in range(n):
        S = d * S + k[t][:, :, None] * v[t][:, None, :]
        out.append((q[t][:, :, None] * S).sum(1))
    o = torch.stack(out)
    o = o / torch.sqrt((o * o).mean(-1, keepdim=True) + eps)
    return o.reshape(n, hv) * gate * torch.sigmoid(gate), S


def _ratio(a, b):
    return float((a.double() - b).norm() / b.norm())


# Rows of ordinary size, and queries, keys and values times powers of two that leave the products where they were: numbers whose bf16 parts
# would fall below bf16's smallest, scores beyond 2^79, a fresh and a carried state.  Tolerance: decays by powf (two units in the last
# place), some 200 rounded products of random signs, the norm and the gate: 2e-6 is ten times what they add up to.
@pytest.mark.parametrize("n,dim,vdim", [(128, 64, 128), (300, 64, 128), (131, 8, 72), (257, 40, 128)])
@pytest.mark.parametrize("pos", [0, 37])
@pytest.mark.parametrize("xq,xk,xv", [(0, 0, 0), (58, -118, 60), (-20, -100, 120), (60, 60, -120), (26, -126, 100)])
def test_retention_in_pieces_of_128_against_float64(n, dim, vdim, pos, xq, xk, xv):
    from umbrella_b200 import ops_seq as K
    heads = 2
    x = torch.randn(n, 2 * heads * (dim + vdim), generator=torch.Generator().manual_seed(n)).to(DEV)
    hd = heads * dim
    x[:, :hd] *= 2.0 ** xq
    x[:, hd:2 * hd] *= 2.0 ** xk
    x[:, 2 * hd:2 * hd + heads * vdim] *= 2.0 ** xv
    decay = torch.tensor([0.93, 0.9995], device=DEV)
    state = torch.randn(1, heads, dim, vdim, generator=torch.Generator().manual_seed(1)).to(DEV) * 2.0 ** (xk + xv)
    want, S = _retention64(x, heads, dim, vdim, decay, state[0] * (pos > 0), 1e-6)
    got = K.retention(x, K.RaggedBatch([(0, n, pos, 0)], DEV), heads, dim, vdim, 0, torch.zeros(1, device=DEV), decay, 1e-6, state, k_scale=1.0)
    assert _ratio(got, want) < 2e-6 and _ratio(state[0], S) < 2e-6


def test_gates_of_pieces_of_128_over_their_range():
    """Row by row, from gates whose silu is near the smallest normal number (there 1 + e^-g is beyond 2^126) up to ordinary ones.  Tolerance as above."""
    from umbrella_b200 import ops_seq as K
    n, heads, dim, vdim = 130, 2, 64, 128
    x = torch.randn(n, 2 * heads * (dim + vdim), generator=torch.Generator().manual_seed(2)).to(DEV)
    x[:, -heads * vdim:] = torch.linspace(-88.5, 3.0, n, device=DEV)[:, None]
    decay, state = torch.tensor([0.93, 0.9995], device=DEV), torch.zeros(1, heads, dim, vdim, device=DEV)
    want, _ = _retention64(x, heads, dim, vdim, decay, state[0], 1e-6)
    got = K.retention(x, K.RaggedBatch([(0, n, 0, 0)], DEV), heads, dim, vdim, 0, torch.zeros(1, device=DEV), decay, 1e-6, state, k_scale=1.0).double()
    assert float(((got - want).norm(dim=1) / want.norm(dim=1)).max()) < 2e-6
