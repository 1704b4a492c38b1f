// What the matrix-product kernels of the sequence-state decoders share: the argument block and what happens to a sum.
#pragma once
#include "seq_internal.h"

namespace umbs {

struct GemmArgs {
    const void* A; int64_t lda; int a_goff;
    const void* W; int64_t ldw; int64_t w_gstride;
    void* C; int64_t ldc; int c_goff;
    int M, N, K;
    const int32_t* grp_off;
    const int32_t* row_src;
    float limit;
    int act;          // UMBS_ACT_*: which gated activation a dual product applies
    const float* bias;       // fp32 [N] (dual: [2 N]) added to the sums, or NULL
    const float* out_gate;   // fp32: the result is multiplied by sigmoid(out_gate[row ld_gate + g gate_goff + n]), or NULL
    int64_t ld_gate;
    int gate_goff;
    int gate_n;       // 1: a gate per output element, 0: one per row and group
    int unary;        // UMBS_UNARY_* of a plain product's first unary_cols columns, with its two numbers
    float p0, p1;
    int unary_cols;
    int rows_total;          // of C, rows sorted by group: those of no group are set to zero (0: not asked for)
    int weights_ready;       // W was there before the chain of launches began: it may be read ahead of chain_wait
};

__device__ __forceinline__ float unary_act(float z, int unary, float p0, float p1) {
    if (unary == UMBS_UNARY_TANH) return tanhf(z);
    if (unary == UMBS_UNARY_XIELU) return z > 0.f ? fmaf(p0 * z, z, 0.5f * z) : fmaf(p1, expm1f(z) - z, 0.5f * z);
    if (unary == UMBS_UNARY_RELU2) { const float r = fmaxf(z, 0.f); return r * r; }
    if (unary == UMBS_UNARY_SILU) return z * (1.f / (1.f + expf(-z)));
    if (unary == UMBS_UNARY_SCALE) return p0 * z;
    return z;
}

__device__ __forceinline__ float gated_act(float g, float u, float limit, int act) {
    if (act == UMBS_ACT_GELU_TANH) {      // 0.5 g (1 + tanh(sqrt(2 / pi) (g + 0.044715 g^3))) * u
        const float z = 0.7978845608028654f * (g + 0.044715f * g * g * g);
        return 0.5f * g * (1.f + tanhf(z)) * u;
    }
    if (act == UMBS_ACT_SILU) return g * (1.f / (1.f + expf(-g))) * u;
    g = fminf(g, limit);
    u = fminf(fmaxf(u, -limit), limit);
    return g * (1.f / (1.f + expf(-1.702f * g))) * (u + 1.f);
}

// What every kernel does with a finished sum (and, for a gate|up pair, its partner): bias and activation ...
template <bool DUAL>
__device__ __forceinline__ float finish_sum(const GemmArgs& a, float s, float s2, int n) {
    if (a.bias != nullptr) {
        s += a.bias[n];
        if (DUAL) s2 += a.bias[a.N + n];
    }
    return DUAL ? gated_act(s, s2, a.limit, a.act) : (a.unary && n < a.unary_cols ? unary_act(s, a.unary, a.p0, a.p1) : s);
}
// ... then the output gate.
__device__ __forceinline__ float finish_gate(const GemmArgs& a, float v, int g, int64_t row, int n) {
    return a.out_gate == nullptr ? v : v * (1.f / (1.f + expf(-a.out_gate[row * a.ld_gate + (int64_t)g * a.gate_goff + n * a.gate_n])));
}
template <bool DUAL>
__device__ __forceinline__ float finish(const GemmArgs& a, float s, float s2, int g, int64_t row, int n) {
    return finish_gate(a, finish_sum<DUAL>(a, s, s2, n), g, row, n);
}

// seq_gemm_tc.cu: bf16 operands, 16-byte rows (the caller has checked them)
int launch_gemm_tc(const GemmArgs& a, int groups, bool dual, bool c_f32, cudaStream_t st);
int tc_tile_columns(int M, int N, int K, int groups, bool dual, bool by_group, bool gathered, int sms);     // columns of its tiles, or UMBS_GEMM_PAIRS
// seq_gemm_split.cu: fp32 operands, 16-byte rows, K a multiple of 4 (the caller has checked them)
int launch_gemm_split(const GemmArgs& a, int groups, bool dual, cudaStream_t st);

}  // namespace umbs
