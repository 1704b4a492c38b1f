"""What a decode step reads of a cache: means of whole blocks (umbs_kv_pool) bit for bit, the routing of up to 148 tokens bit for bit, and the grouped attention with four and with six warps
a block (unsplit steps from 148 blocks on) against float64.

Tolerance: results are bf16 (2^-9 of their size at most, 2^-9 / sqrt(3) in the norm); the fp32 work inside is four orders below."""
import ctypes as C

import pytest
import torch

import seq_helpers as H

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("row", [8, 12, 136, 264])                                   # one piece; no whole pieces; a tail behind 128 columns
@pytest.mark.parametrize("pool,pos0,tokens,kv_len", [(1, 3, 2, 8), (16, 15, 1, 40), (7, 20, 40, 50), (8, 20, 40, 50), (33, 30, 80, 64), (64, 63, 1, 64), (64, 70, 130, 90), (100, 150, 60, 128)])
def test_means_of_blocks(dt, row, pool, pos0, tokens, kv_len):
    from umbrella_b200 import _lib_seq as S, ops_seq as K
    g = torch.Generator().manual_seed(7)
    kv, ring = (torch.randn(*s, generator=g).to(dt) for s in ((2 * tokens, row), (3, kv_len, row)))
    blocks = (pos0 + tokens) // pool + 1
    b = K.RaggedBatch([(2, tokens, pos0, 0), (0, tokens, pos0, 0)], DEV)
    d_kv, d_ring, means = kv.to(DEV), ring.to(DEV), torch.full((3, blocks, row), 5.0, dtype=dt, device=DEV)
    S.check(S.load().umbs_kv_pool(S.UMBS_BF16 if dt == torch.bfloat16 else S.UMBS_F32, d_kv.data_ptr(), d_ring.data_ptr(), kv_len, means.data_ptr(), blocks,
                                  C.byref(b.c), row, pool, torch.cuda.current_stream().cuda_stream), "kv_pool")
    want = torch.full((3, blocks, row), 5.0, dtype=dt)
    for s, slot in enumerate((2, 0)):
        for blk in range(pos0 // pool, (pos0 + tokens) // pool):
            acc = torch.zeros(row)
            for j in range(blk * pool, (blk + 1) * pool):
                acc += (kv[s * tokens + j - pos0] if j >= pos0 else ring[slot, j % kv_len]).float()
            want[slot, blk] = (acc / torch.tensor(float(pool))).to(dt)
    assert torch.equal(means.cpu(), want)


@pytest.mark.parametrize("mode", ["SOFTMAX", "SOFTMAX_SINK", "SIGMOID"])
@pytest.mark.parametrize("seqs,kv_heads,group,dim,ctx", [(37, 4, 2, 64, 230), (36, 4, 2, 64, 230), (148, 1, 9, 40, 193), (150, 1, 3, 128, 33), (75, 2, 4, 96, 400)])
def test_groups_of_heads(mode, seqs, kv_heads, group, dim, ctx):
    from umbrella_b200 import _lib_seq as S, ops_seq as K
    g = torch.Generator(device=DEV).manual_seed(8)
    r = lambda *s: torch.randn(*s, generator=g, device=DEV).bfloat16()
    heads, row = kv_heads * group, 2 * kv_heads * dim
    pos = [max(0, ctx - 1 - 7 * (i % 5)) for i in range(seqs)]
    q, kv, cache, sink = r(seqs, heads * dim), r(seqs, row), r(seqs, ctx + 3, row), r(heads).float()
    b = K.RaggedBatch([(i, 1, p, 0) for i, p in enumerate(pos)], DEV)
    out = K.cached_attention(q, kv, cache.clone(), b, heads, kv_heads, dim, dim, dim ** -0.5, mode=getattr(S, "UMBS_ATTN_" + mode), sink=sink if "SINK" in mode else None)
    for i in range(0, seqs, 7):
        rows = torch.cat([cache[i, :pos[i]], kv[i:i + 1]]).double().view(pos[i] + 1, 2, kv_heads, dim)
        z = torch.einsum("hgd,jhd->hgj", q[i].double().view(kv_heads, group, dim), rows[:, 0]) * dim ** -0.5
        if mode == "SIGMOID":
            w = torch.sigmoid(z)
        else:
            e = torch.cat([z, sink.double().view(kv_heads, group, 1)], 2) if "SINK" in mode else z
            w = torch.softmax(e, 2)[..., :pos[i] + 1]
        want = torch.einsum("hgj,jhd->hgd", w, rows[:, 1]).reshape(-1)
        assert H.rel_err(out[i], want) < 2.0 ** -9


@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("n,experts,width,top,gate", [(17, 15, 100, 2, True), (17, 16, 1024, 3, False), (64, 16, 1152, 2, True), (64, 17, 2052, 1, False), (64, 300, 64, 9, True),
                                                      (20, 1024, 1030, 4, False), (20, 1025, 128, 4, False), (148, 8, 1152, 2, False), (148, 130, 512, 6, True)])
def test_routing_of_few_tokens(dt, n, experts, width, top, gate):
    """A block to a token and warps with one or two experts choose what four tokens to a block and four experts to a warp do (the same tokens among 170)."""
    from umbrella_b200 import _lib_seq as S, ops_seq as K
    g = torch.Generator().manual_seed(9)
    h, w, gw = torch.randn(170, width, generator=g).to(dt).to(DEV), torch.randn(experts, width, generator=g).to(DEV), torch.randn(width, generator=g).to(DEV)
    few, many = (K.moe_route_ex(h[:m], w, top, S.UMBS_ROUTE_SOFTMAX_TOP, gate_w=gw if gate else None) for m in (n, 170))
    for i in [0, 4] + [5] * gate:
        assert torch.equal(few[i], many[i][:n])
    off, tok, pos, sel = (t.cpu() for t in few[1:5])
    assert torch.equal(off, torch.cat([torch.zeros(1), torch.bincount(sel.flatten().long(), minlength=experts).cumsum(0)]).int())
    place = pos.view(n, top).long()
    assert torch.equal(tok[place], torch.arange(n, dtype=torch.int32)[:, None].expand(n, top)) and torch.equal(place.flatten().sort().values, torch.arange(n * top))
    assert bool(((place >= off[sel.long()]) & (place < off[sel.long() + 1])).all())
