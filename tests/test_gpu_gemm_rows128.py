"""The AWQ product with 33 to 128 token rows, where the head of a split tile is reduced by all groups of warps in turn, and
beyond 64 rows with weight records and x slabs in rings of their own (csrc/gemm.cu, kSplit).  K from one unit of 128 (fewer units than a ring is deep) to many tiles a
block shares, rows at the edges of the 16-row chunks, every epilogue that stages rows."""
import numpy as np
import pytest
import torch

from oracle import awq as oawq

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _near(out, ref, slack):
    """fp16 results round once or twice (2^-11 of the value each); `slack` bounds the fp32 sums' own error."""
    err = (out.double().cpu() - ref).abs()
    return bool((err <= 2.0 ** -10 * ref.abs() + slack).all())


@pytest.mark.parametrize("M,K,N", [(65, 128, 128), (80, 512, 640), (81, 4096, 4096), (112, 14336, 512), (113, 1024, 2048),
                                   (127, 2048, 128), (128, 4096, 6144), (33, 4096, 4096), (49, 1024, 640), (64, 14336, 512)])
def test_rows_33_to_128(M, K, N):
    from umbrella_b200 import ops
    rng = np.random.default_rng(M + K + N)
    packed = ops.awq_repack(*(torch.from_numpy(t).to(DEV) for t in oawq.random_awq(K, N, 128, rng)))
    x = torch.from_numpy((rng.standard_normal((M, K)) * 0.5).astype(np.float16)).to(DEV)
    res = torch.from_numpy(rng.standard_normal((M, N)).astype(np.float16)).to(DEV)
    ws = ops.gemm_workspace(M, K, N, DEV)
    w = ops.awq_unpack(packed, K, N).double().cpu()                      # [N, K]: the fp16 weights the kernel multiplies
    xd = x.double().cpu()
    y = xd @ w.t()
    slack = K * 2.0 ** -24 * (xd.abs() @ w.abs().t())
    out = ops.awq_gemm(x, packed, K, N, workspace=ws)
    assert _near(out, y, slack)
    y16 = out.double().cpu()                                             # the rounded product, then one rounded sum
    outr = res.clone()
    ops.awq_gemm(x, packed, K, N, mode=ops.UMB_EPI_RESIDUAL, residual=outr, out=outr, workspace=ws)
    assert torch.equal(outr.cpu(), (y16 + res.double().cpu()).to(torch.float16))
    outs = ops.awq_gemm(x, packed, K, N, mode=ops.UMB_EPI_SILU_MUL, workspace=ws)
    gate, up = y16.view(M, N // 128, 2, 64).unbind(2)
    s = (gate * torch.sigmoid(gate)).reshape(M, N // 2)
    ref = s * up.reshape(M, N // 2)
    assert _near(outs, ref, 1e-6 + 2.0 ** -10 * ref.abs())               # silu and the product round on their own
    for _ in range(5):
        assert torch.equal(ops.awq_gemm(x, packed, K, N, workspace=ws), out)
    assert int(ws.view(torch.int32).abs().max()) == 0                    # the workspace is handed on clean


@pytest.mark.parametrize("M", [33, 49, 64, 65, 128])
def test_rope_rows_33_to_128(M):
    """The rotary epilogue stages its output and the rows of cos and sin in each group's own rows: the bits of the product followed by
    umb_rope_append_f16, with K long enough that tiles are split over blocks."""
    from umbrella_b200 import ops
    Hq, Hkv, D, K, S, off = 16, 4, 128, 4096, 256, 77
    rng = np.random.default_rng(M)
    N = (Hq + 2 * Hkv) * D
    x = torch.from_numpy((rng.standard_normal((M, K)) * 0.5).astype(np.float16)).to(DEV)
    packed = ops.awq_repack(*(torch.from_numpy(t).to(DEV) for t in oawq.random_awq(K, N, 128, rng, scale=0.02)))
    pos = torch.from_numpy(rng.integers(0, S, M)).to(DEV)
    ang = torch.rand(S, D, device=DEV) * 6.28
    cos, sin = ang.cos().to(torch.float16), ang.sin().to(torch.float16)
    outs = []
    for fused in (False, True):
        q = torch.zeros(M, Hq, D, dtype=torch.float16, device=DEV)
        k = torch.zeros(S, Hkv, D, dtype=torch.float16, device=DEV)
        v = torch.zeros_like(k)
        if fused:
            rope = ops.make_rope_epilogue(q, k, v, cos, sin, pos, Hq, Hkv, D, off)
            ops.awq_gemm(x, packed, K, N, mode=ops.UMB_EPI_ROPE_QKV, rope=rope, out=torch.zeros(M, N, dtype=torch.float16, device=DEV))
        else:
            ops.rope_append(ops.awq_gemm(x, packed, K, N), q, k, v, cos, sin, pos, Hq, Hkv, D, off)
        outs.append((q, k, v))
    for a, b in zip(*outs):
        assert torch.equal(a, b)
    assert outs[1][1][off:off + M].abs().sum() > 0


@pytest.mark.parametrize("M", [33, 64, 65, 128])
def test_logits_with_their_largest_rows_33_to_128(M):
    """The fp32 results of an AWQ head are the fp16 products' numbers, and the keys name each row's largest."""
    from umbrella_b200 import ops
    K, N = 4096, 3072
    rng = np.random.default_rng(M)
    packed = ops.awq_repack(*(torch.from_numpy(t).to(DEV) for t in oawq.random_awq(K, N, 128, rng, scale=0.02)))
    x = torch.from_numpy((rng.standard_normal((M, K)) * 0.5).astype(np.float16)).to(DEV)
    keys = torch.zeros(M, dtype=torch.int64, device=DEV)
    logits = ops.awq_gemm(x, packed, K, N, mode=ops.UMB_EPI_LOGITS, argmax=keys)
    assert logits.dtype == torch.float32 and torch.equal(logits, ops.awq_gemm(x, packed, K, N).float())
    assert torch.equal(ops.argmax_keys_to_ids(keys).cpu(), logits.cpu().argmax(-1))


@pytest.mark.parametrize("M", [65, 100, 128])
def test_sums_as_good_as_those_of_fewer_rows(M):
    """A tile's k goes into two accumulators whatever its rows are, which the tensor core cuts off at each of half as many steps as one would take.  What that
    leaves shows in how many results are not the float64 product rounded: as many as when the same rows are multiplied 64 at a time (half of one per cent
    here; one accumulator: 1.8 times that).  A tenth more is four standard deviations of the count."""
    from umbrella_b200 import ops
    K, N = 14336, 4096
    rng = np.random.default_rng(M)
    packed = ops.awq_repack(*(torch.from_numpy(t).to(DEV) for t in oawq.random_awq(K, N, 128, rng)))
    x = torch.from_numpy((rng.standard_normal((M, K)) * 0.5).astype(np.float16)).to(DEV)
    want = (x.double() @ ops.awq_unpack(packed, K, N).double().t()).to(torch.float16)
    few = torch.cat([ops.awq_gemm(x[i:i + 64], packed, K, N) for i in range(0, M, 64)])
    off = [int((y != want).sum()) for y in (ops.awq_gemm(x, packed, K, N), few)]
    assert 0 < off[0] < 1.1 * off[1] + 50, off
