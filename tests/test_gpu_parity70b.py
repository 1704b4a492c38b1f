"""GPU parity at the headline shape: the native verify forward at Llama-3.1-70B dimensions
(H = 8192, I = 28672, 64 / 8 heads, V = 128256) against

  (b) the fp32 oracle (oracle/llama.py: the reference's op order, fp32 maths, the reference's fp16 rounding
      points), streamed layer by layer on the device -- the 80-layer model does not fit a CPU run in seconds; and
  (c) the reference's own kernels on the same inputs (tests/refkernels.py: vLLM's build of the upstream AWQ GEMM,
      flashinfer single_prefill_with_kv_cache(custom_mask) and flashinfer.rmsnorm, glued as llama.py:262-322).

Tolerance: logits within 1e-3, read relative to max|logit| -- or, where the reference's own
kernels sit farther than that from the fp32 oracle, the measured reference noise (both distances are
printed).

Also here: every fused full-width GEMM of a 70B layer (q|k|v N = 10240, gate|up N = 57344 with the SiLU epilogue,
o, down) against the oracle's dequantiser (validated against the numpy oracle on CPU), not against the kernel's
own unpack.
"""
import json
import os

import numpy as np
import pytest
import torch

from oracle import awq as oawq
from oracle import llama as ollama
from oracle import tree as otree

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
GOLDEN = os.path.join(os.path.dirname(__file__), "golden")
TOL = 1e-3                      # target logits match the reference within 1e-3 (fp16)


def _tree():
    trees = json.load(open(os.path.join(GOLDEN, "trees.json")))["shipped"]
    return otree.growmap_from_successors(trees["sequoia_tree-3x4.json"]["Successors"])


def _rel(a, ref):
    return float((a.double() - ref.double()).abs().max() / ref.double().abs().max())


@pytest.mark.parametrize("layers", [8, 80])
def test_70b_shape_logits_vs_oracle_and_reference_kernels(layers):
    import refkernels
    from umbrella_b200.models import llama as L
    shape, S, P, seed = L.LLAMA31_70B, 256, 48, 2024
    oshape = ollama.LLAMA31_70B
    gm = _tree()
    tm = np.asarray(gm["mask"], dtype=bool)
    N, depth = gm["size"], np.asarray(gm["depth"])
    g = torch.Generator().manual_seed(layers)
    prompt = torch.randint(3, shape.vocab_size, (1, P), generator=g).to(DEV)
    tree_tokens = torch.randint(3, shape.vocab_size, (1, N), generator=g).to(DEV)
    pos_p = torch.arange(P, device=DEV)[None]
    pos_t = (P + torch.from_numpy(depth)).to(DEV)[None]
    causal = torch.from_numpy(otree.make_causal_mask(P)).to(DEV)
    dense = torch.from_numpy(otree.dense_rows_from_compact(P, tm, P + N)).to(DEV)

    model = L.LlamaAwq(shape, max_length=S, device=DEV, num_layers=layers)
    model.alloc()
    res = refkernels.three_way_logits(L, ollama, shape, oshape, True, seed, layers, prompt, tree_tokens, pos_p, pos_t, causal,
                                      dense, model.cos_cache, model.sin_cache, DEV, on_layer=model.load_awq_layer, max_length=S)
    head = res["head"]
    model.load_head(head["embed_tokens"], head["lm_head"], head["norm"])
    o16, ox, ref_why = res["oracle"], res["oracle_exact"], res["reference_unavailable"]

    model.inference(prompt, pos_p, causal)
    ours = model.inference(tree_tokens, pos_t, dense)[0]
    torch.cuda.synchronize()

    rec = {"layers": layers, "prompt_rows": P, "tree_rows": N, "max_abs_logit": float(o16.abs().max()),
           "ours_vs_fp32_oracle": _rel(ours, o16), "ours_vs_exact_weight_oracle": _rel(ours, ox),
           "oracle_fp16w_vs_exact": _rel(o16, ox)}
    if ref_why is None:
        ref = res["reference"]
        rec.update(reference_kernels_vs_fp32_oracle=_rel(ref, o16), reference_kernels_vs_exact_weight_oracle=_rel(ref, ox),
                   ours_vs_reference_kernels=_rel(ours, ref),
                   reference_kernels="vLLM 0.22 _C.awq_gemm(split_k_iters=8) + flashinfer 0.6.11 single_prefill_with_kv_cache("
                                     "custom_mask, fp32 QK reduction) + flashinfer.rmsnorm")
    else:
        rec["reference_kernels_unavailable"] = ref_why
    print("\nparity70b", json.dumps(rec))

    # yardstick: the fp32 oracle with the reference's rounding points (fp16-rounded weights, as both the upstream kernel
    # and the product feed their MMAs); bar: the 1e-3 that is asked for or, where the reference's own kernels sit farther than that
    # from the same oracle, their measured distance.  (The exact-weight oracle's distances are in the record too.)
    bound = max(TOL, rec.get("reference_kernels_vs_fp32_oracle", 0.0))
    assert rec["ours_vs_fp32_oracle"] <= bound, rec
    # arg-max equal wherever the oracle's top-2 margin exceeds twice the bound
    top2 = o16.topk(2, dim=-1).values
    safe = (top2[:, 0] - top2[:, 1]) > 2 * bound * o16.abs().max()
    assert torch.equal(ours.argmax(-1)[safe], o16.argmax(-1)[safe])


def _gemm_ref(x, triplet, exact=False):
    w = oawq.dequantize_torch(*triplet, 128, exact=exact).double()
    return (x.double() @ w).to(torch.float16)


@pytest.mark.parametrize("M", [13, 31])
def test_70b_full_width_gemms_vs_oracle(M):
    """The four fused AWQ streams of one 70B layer at their real widths against x @ fp16((q - z) * s) in float64."""
    from umbrella_b200 import ops
    from umbrella_b200.models import llama as L
    shape = L.LLAMA31_70B
    H, I = shape.hidden_size, shape.intermediate_size
    raw = L.synth_layer(shape, 0, True, 99, gen_device=DEV)
    g = torch.Generator(device=DEV).manual_seed(M)
    x = torch.randn(M, H, generator=g, device=DEV).to(torch.float16)
    xi = (0.05 * torch.randn(M, I, generator=g, device=DEV)).to(torch.float16)
    nq, nkv = H, shape.num_key_value_heads * shape.head_dim
    # q|k|v: one stream, N = 10240
    qkv_n = nq + 2 * nkv
    wqkv = ops.awq_repack(*raw["wq"], N_total=qkv_n)
    ops.awq_repack(*raw["wk"], packed=wqkv, N_total=qkv_n, row_offset=nq)
    ops.awq_repack(*raw["wv"], packed=wqkv, N_total=qkv_n, row_offset=nq + nkv)
    out = ops.awq_gemm(x, wqkv, H, qkv_n)
    ref = torch.cat([_gemm_ref(x, raw[n]) for n in ("wq", "wk", "wv")], dim=1)
    assert _rel(out, ref) < TOL
    # o with the residual epilogue, N = 8192
    res = torch.randn(M, H, generator=g, device=DEV).to(torch.float16)
    out = ops.awq_gemm(x, ops.awq_repack(*raw["wo"]), H, H, mode=ops.UMB_EPI_RESIDUAL, residual=res)
    assert _rel(out, res + _gemm_ref(x, raw["wo"])) < 2 * TOL
    # gate|up with the SiLU epilogue, N = 57344 -> 28672 outputs
    wgu = ops.awq_repack(*raw["gate_proj"], N_total=2 * I, row_block=64, row_stride=128)
    ops.awq_repack(*raw["up_proj"], packed=wgu, N_total=2 * I, row_block=64, row_stride=128, row_offset=64)
    out = ops.awq_gemm(x, wgu, H, 2 * I, mode=ops.UMB_EPI_SILU_MUL)
    gate = torch.nn.functional.silu(_gemm_ref(x, raw["gate_proj"]).float()).to(torch.float16)
    ref = gate * _gemm_ref(x, raw["up_proj"])
    assert out.shape == (M, I)
    assert _rel(out, ref) < 3 * TOL                 # two fp16 roundings (silu, product) on top of the GEMM's
    # down, K = 28672
    out = ops.awq_gemm(xi, ops.awq_repack(*raw["down_proj"]), I, H, mode=ops.UMB_EPI_RESIDUAL, residual=res)
    assert _rel(out, res + _gemm_ref(xi, raw["down_proj"])) < 2 * TOL
