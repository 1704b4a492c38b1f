"""Attention of many query rows (64-row tiles, weights in two fp16 parts) against float64, on both sides of the line to the slabs of 16 rows (128 tiles
over all key/value heads) and at the edges of its tiles.

Tolerance: results are fp16, 2^-11 of their size at most and 2^-11 / sqrt(3) = 2.8e-4 in the norm; the two parts leave 2^-22 of a weight, one part (the
slabs) 2^-12 / sqrt(3) = 1.4e-4: together 3.2e-4."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("mode", ["causal", "tree", "dense"])
@pytest.mark.parametrize("qo,prefix,heads,kv_heads,dim,cap", [(256, 0, 32, 8, 128, 0.0), (240, 70, 32, 8, 128, 0.0), (241, 70, 32, 8, 128, 0.0), (505, 3, 16, 16, 64, 0.0),
                                                             (130, 500, 64, 8, 64, 30.0), (333, 1, 24, 8, 128, 20.0)])
def test_many_rows(mode, qo, prefix, heads, kv_heads, dim, cap):
    from umbrella_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(5)
    kv, G = prefix + qo, heads // kv_heads
    r = lambda *s: torch.randn(*s, generator=g, device=DEV).half()
    q, k, v = r(qo, heads, dim), r(kv + 9, kv_heads, dim), r(kv + 9, kv_heads, dim)
    i, j = torch.arange(qo, device=DEV)[:, None], torch.arange(kv, device=DEV)[None]
    if mode == "causal":
        see, mask = j <= prefix + i, ops.make_mask(2, prefix)
    elif mode == "tree":
        bits = torch.rand(qo, qo, generator=g, device=DEV) < 0.3
        bits.fill_diagonal_(True)
        words = torch.zeros(qo, (qo + 31) // 32 * 32, dtype=torch.int64, device=DEV)
        words[:, :qo] = bits
        words = (words.view(qo, -1, 32) << torch.arange(32, device=DEV)).sum(-1)
        words = torch.where(words >= 1 << 31, words - (1 << 32), words).int().contiguous()
        see, mask = torch.cat([torch.ones(qo, prefix, dtype=torch.bool, device=DEV), bits], 1), ops.make_mask(0, prefix, tree_bits=words)
    else:
        see = torch.rand(qo, kv, generator=g, device=DEV) < 0.5
        see[:, 0] = True
        dense = see.to(torch.uint8).contiguous()
        mask = ops.make_mask(1, prefix, dense_mask=dense)
    out = ops.tree_attn(q, k, v, kv, mask, soft_cap=cap)
    z = torch.einsum("qhd,khd->hqk", q.double(), k[:kv].double().repeat_interleave(G, 1)) * dim ** -0.5
    if cap:
        z = cap * torch.tanh(z / cap)
    want = torch.einsum("hqk,khd->qhd", torch.softmax(z.masked_fill(~see, -torch.inf), -1), v[:kv].double().repeat_interleave(G, 1))
    assert float((out.double() - want).norm() / want.norm()) < 3.2e-4
