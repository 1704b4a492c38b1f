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
