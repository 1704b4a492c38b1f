"""Attention of many query rows against float64: tiles of 64 rows with weights in two fp16 parts (csrc/attn_rules.h says when) and slabs of 16 rows beside them, at the edges
of both.

Tolerance: a result is rounded to fp16, which leaves 2^-11 / sqrt(3) of its binade and 2.03e-4 in the norm of results of all sizes; two parts leave 2^-22 of a weight,
nothing to that, one part (the slabs) 2^-12 / sqrt(3) = 1.4e-4 of each: in all 2.46e-4 where a row's weights are of all sizes.  So tiles stay below 2.25e-4,
which one part would pass, slabs below 3.2e-4."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("mode", ["causal", "tree", "dense"])
@pytest.mark.parametrize("qo,prefix,heads,kv_heads,dim,cap,tiled", [(256, 0, 32, 8, 128, 0.0, "causal"), (240, 70, 32, 8, 128, 0.0, ""), (241, 70, 32, 8, 128, 0.0, "causal"),
                                                                   (505, 3, 16, 16, 64, 0.0, ""), (130, 500, 64, 8, 64, 30.0, ""), (333, 1, 24, 8, 128, 20.0, "causal"),
                                                                   (300, 500, 64, 8, 128, 0.0, "causal tree"), (257, 300, 64, 8, 128, 20.0, "causal tree"),
                                                                   (300, 0, 32, 8, 64, 0.0, "causal"), (200, 80, 64, 8, 64, 30.0, "causal")])
def test_many_rows(mode, qo, prefix, heads, kv_heads, dim, cap, tiled):
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
    assert float((out.double() - want).norm() / want.norm()) < (2.25e-4 if mode in tiled else 3.2e-4)
