"""What a decode step reads of a cache: means of whole blocks (umbs_kv_pool), bit for bit."""
import ctypes as C

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("row", [8, 12, 136, 264])                                   # one piece; no whole pieces; a tail behind 128 columns
@pytest.mark.parametrize("pool,pos0,tokens,kv_len", [(1, 3, 2, 8), (16, 15, 1, 40), (64, 63, 1, 64), (64, 70, 130, 90), (100, 150, 60, 128)])
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
