"""AWQ products of up to 512 token rows.  By pairs of SMs (from 129 rows on): tiles held by one pair, shared by two and by many, an odd number of tiles (the
second block of the last pair of tiles has none), fewer k units than a ring is deep, both sides of every accumulator width and of the
step to two blocks of rows, and of the step to that kernel; the longest sums, which go in passes.

Tolerance of sums: an accumulator is cut off behind every 16 of k, by 2^-23 of itself at most, and the parts of a tile are added with as much; it is seldom more than six
times what the root of the summed squares of the products makes it.  (K 2^-24 of the summed sizes, as a bound for any order, would be 6 % of a result of 14336.)"""
import ctypes as C

import numpy as np
import pytest
import torch

from oracle import awq as oawq

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _run(x, packed, K, N, ws, mode=0, residual=None, rope=None, argmax=None, out=None):
    from umbrella_b200 import _lib, ops
    M, n_out = x.shape[0], N // 2 if mode == ops.UMB_EPI_SILU_MUL else N
    if out is None:
        out = torch.empty(M, n_out, dtype=torch.float32 if mode == ops.UMB_EPI_LOGITS else torch.float16, device=DEV)
    e = ops._epilogue(mode, None, residual, argmax, rope)
    _lib.check(_lib.load().umb_awq_gemm_rows_f16(x.data_ptr(), x.stride(0), packed.data_ptr(), out.data_ptr(), out.stride(0), M, K, N, 128, C.byref(e),
                                                 ws.data_ptr(), ws.numel(), torch.cuda.current_stream().cuda_stream), "rows")
    return out


def _setup(M, K, N, scale=0.003):
    from umbrella_b200 import _lib, ops
    rng = np.random.default_rng(M + K + N)
    packed = ops.awq_repack(*(torch.from_numpy(t).to(DEV) for t in oawq.random_awq(K, N, 128, rng, scale=scale)))
    x = torch.from_numpy((rng.standard_normal((M, K)) * 0.5).astype(np.float16)).to(DEV)
    ws = torch.zeros(_lib.load().umb_awq_gemm_rows_ws_bytes(M, K, N), dtype=torch.uint8, device=DEV)
    return packed, x, ws


def _near(out, ref, slack):
    """fp16 results round once or twice (2^-11 of the value each); `slack` bounds the fp32 sums' own error."""
    return bool(((out.double() - ref).abs() <= 2.0 ** -10 * ref.abs() + slack).all())


@pytest.mark.parametrize("M,K,N", [(65, 128, 384), (128, 4096, 28672), (129, 128, 128), (192, 640, 1152), (193, 4096, 4096), (256, 14336, 512),
                                   (257, 4096, 6144), (300, 384, 19072), (384, 2048, 640), (385, 4096, 1024), (500, 4096, 28672), (512, 1024, 2304)])
def test_rows_up_to_512(M, K, N):
    from umbrella_b200 import ops
    packed, x, ws = _setup(M, K, N)
    res = torch.randn(M, N, device=DEV).to(torch.float16)
    w, xd = ops.awq_unpack(packed, K, N).double(), x.double()
    y = xd @ w.t()
    slack = (K / 16 + 8) * 2.0 ** -23 * 6 * ((xd * xd) @ (w * w).t()).sqrt()
    out = _run(x, packed, K, N, ws)
    assert _near(out, y, slack)
    y16 = out.double()
    outr = res.clone()
    _run(x, packed, K, N, ws, mode=ops.UMB_EPI_RESIDUAL, residual=outr, out=outr)
    assert torch.equal(outr, (y16 + res.double()).to(torch.float16))
    gate, up = y16.view(M, N // 128, 2, 64).unbind(2)
    ref = (gate * torch.sigmoid(gate) * up).reshape(M, N // 2)
    assert _near(_run(x, packed, K, N, ws, mode=ops.UMB_EPI_SILU_MUL), ref, 1e-6 + 2.0 ** -10 * ref.abs())      # silu and the product round on their own
    keys = torch.zeros(M, dtype=torch.int64, device=DEV)
    logits = _run(x, packed, K, N, ws, mode=ops.UMB_EPI_LOGITS, argmax=keys)
    assert torch.equal(logits, out.float()) and torch.equal(ops.argmax_keys_to_ids(keys), logits.argmax(-1))
    for _ in range(5):
        assert torch.equal(_run(x, packed, K, N, ws), out)
    assert int(ws.view(torch.int32).abs().max()) == 0                    # the workspace is handed on clean


@pytest.mark.parametrize("M,D", [(129, 128), (256, 64), (300, 128)])
def test_rope_rows(M, D):
    """The bits of the product followed by umb_rope_append_f16."""
    from umbrella_b200 import ops
    Hq, Hkv, K, S, off = 16, 4, 2048, 512, 77
    N = (Hq + 2 * Hkv) * D
    packed, x, ws = _setup(M, K, N, scale=0.02)
    pos = torch.randint(0, S, (M,), device=DEV)
    ang = torch.rand(S, D, device=DEV) * 6.28
    cos, sin = ang.cos().to(torch.float16), ang.sin().to(torch.float16)
    outs = []
    for fused in (False, True):
        q = torch.zeros(M, Hq, D, dtype=torch.float16, device=DEV)
        k = torch.zeros(S, Hkv, D, dtype=torch.float16, device=DEV)
        v = torch.zeros_like(k)
        if fused:
            _run(x, packed, K, N, ws, mode=ops.UMB_EPI_ROPE_QKV, rope=ops.make_rope_epilogue(q, k, v, cos, sin, pos, Hq, Hkv, D, off))
        else:
            ops.rope_append(_run(x, packed, K, N, ws), q, k, v, cos, sin, pos, Hq, Hkv, D, off)
        outs.append((q, k, v))
    for a, b in zip(*outs):
        assert torch.equal(a, b)
    assert outs[1][1][off:off + M].abs().sum() > 0


@pytest.mark.parametrize("rows", [129, 500, 513])
def test_passes_of_a_prompt_agree(rows):
    """A prompt through passes of 128 rows and of as many as a pass takes: the same model up to the rounding of its sums, whatever comes last."""
    from umbrella_b200.models import llama
    shape = llama.LlamaShape(hidden_size=512, intermediate_size=1024, num_hidden_layers=2, num_attention_heads=4, num_key_value_heads=2, vocab_size=1000,
                             rope_scaling=None)
    m = llama.SyntheticLlama(shape, max_length=640, awq=True)
    ids, pos = torch.randint(0, 1000, (rows,), device=DEV), torch.arange(rows, device=DEV)
    out = []
    for per_pass in (128, m.rows_per_pass):
        m.clear()
        m.rows_per_pass = per_pass
        out.append((m.prefill_forward(ids, pos, last_only=False), m.k_cache[:, :rows].clone() if m.k_cache.shape[1] >= rows else m.k_cache.clone()))
    (a, ka), (b, kb) = out
    assert float((a - b).norm() / a.norm()) < 4e-3 and float((ka - kb).float().norm() / ka.float().norm()) < 4e-3        # fp16: a few roundings of 2^-11


@pytest.mark.parametrize("M", [13, 64, 100, 300])
def test_silu_rounds_its_quotient(M):
    """fp16(g / (1 + e^-g)) * up with the quotient rounded once in fp32, bit for bit (an approximate reciprocal moves one result in some ten thousand)."""
    from umbrella_b200 import ops
    K, N = 256, 16384
    packed, x, ws = _setup(M, K, N, scale=0.05)
    gate, up = _run(x, packed, K, N, ws).view(M, N // 128, 2, 64).unbind(2)
    g = gate.float()
    want = (g / (1 + torch.exp(-g))).to(torch.float16) * up
    assert torch.equal(_run(x, packed, K, N, ws, mode=ops.UMB_EPI_SILU_MUL), want.reshape(M, N // 2))


@pytest.mark.parametrize("mode", [0, 1, 2, 3])
@pytest.mark.parametrize("M", [129, 300, 512])
def test_the_longest_sums_go_in_passes(M, mode):
    """More than 16384 k: the bits of equal passes of up to 128 rows, whose sums are shorter, with every epilogue's rows where they belong."""
    from umbrella_b200 import ops
    K, N = 16512, 384
    packed, x, ws = _setup(M, K, N)
    res = torch.randn(M, N, device=DEV).to(torch.float16)
    passes = -(-M // 128)
    rows = -(-M // passes)
    keys, want_keys = torch.zeros(M, dtype=torch.int64, device=DEV), torch.zeros(M, dtype=torch.int64, device=DEV)
    logits = mode == ops.UMB_EPI_LOGITS
    want = torch.cat([ops.awq_gemm(x[i:i + rows], packed, K, N, mode=mode, residual=res[i:i + rows] if mode == ops.UMB_EPI_RESIDUAL else None,
                                   argmax=want_keys[i:i + rows] if logits else None) for i in range(0, M, rows)])
    got = _run(x, packed, K, N, ws, mode=mode, residual=res if mode == ops.UMB_EPI_RESIDUAL else None, argmax=keys if logits else None)
    assert torch.equal(got, want) and torch.equal(keys, want_keys)
