"""The AWQ product with 33 to 128 token rows, where the head of a split tile is reduced by all groups of warps in turn, and
beyond 64 rows with weight records and x slabs in rings of their own.  K from one unit of 128 (fewer units than a ring is deep) to many tiles a
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
