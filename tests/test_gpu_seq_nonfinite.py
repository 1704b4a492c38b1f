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
