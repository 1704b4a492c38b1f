// What the attention kernels over a per-slot key/value cache share: arguments, virtual heads, shaped scores.
#pragma once
#include <math.h>

#include "seq_internal.h"

namespace umbs {

struct CachedAttnArgs {
    const void* q; const void* kv; const void* kv_cache; const void* pool_cache;
    int kv_len, pool_len;
    int heads, kv_heads, dim, vdim, window, pool;
    float scale;
    const float* head_bias; const float* gate; int64_t ldg; int gate_per_head;
    void* out;
    // score options
    float softcap; const float* r1; const float* r2; int chunk, maps, vheads; float* raw;
    const float* sink;                                // [heads] or NULL: the sink's score per head (NULL: 0)
};
__device__ __forceinline__ float sink_score(const CachedAttnArgs& a, int h) { return a.sink != nullptr ? a.sink[h] : 0.f; }

// What a virtual head reads: its query's offset in a q row, its keys' and values' offsets in a key/value row.
struct VHead { int h, qoff, koff, voff, row_kv, qstride, nv; };
__device__ __forceinline__ VHead virtual_head(const CachedAttnArgs& a, int vh) {
    const int C = a.vheads, M = a.maps;
    const int cv = vh % C, hm = vh / C, mp = hm % M, h = hm / M, g = h / (a.heads / a.kv_heads);
    const int kdim = a.kv_heads * M * a.dim;
    VHead v;
    v.h = h; v.qoff = hm * a.dim; v.koff = (g * M + mp) * a.dim; v.voff = kdim + (C > 1 ? cv : g) * a.vdim;
    v.row_kv = kdim + a.kv_heads * a.vdim; v.qstride = a.heads * M * a.dim; v.nv = a.heads * M * C;
    return v;
}

// scale, cap and distance penalty of a raw dot product; dist = row position - key position
__device__ __forceinline__ float shaped_score(const CachedAttnArgs& a, float dot, float r1h, float r2h, int dist) {
    float sv = dot * a.scale;
    if (a.softcap > 0.f) sv = a.softcap * tanhf(sv / a.softcap);
    if (a.r1 != nullptr) sv -= r1h * log1pf(r2h * (float)dist);
    return sv;
}

__device__ __forceinline__ float sigmoidf_(float z) { return 1.f / (1.f + expf(-z)); }

// One query row in plain fp32 by a whole warp, a key at a time.  The tensor-core kernels hand a row to it whose result is not
// finite: a key that the row does not see sits in its tile with a weight of 0, and 0 times a NaN value is NaN; the parts that a
// weight is split into are often 0, and 0 times an infinite value is no infinity.  Bound: a load latency per key; it is not there
// for speed.
struct PlainRow { float q[6], o[4], m, l; };          // a lane's numbers: dimensions lane + 32 i (up to 192), value columns (up to 128)
__device__ __forceinline__ void plain_start(PlainRow& s, const __nv_bfloat16* q, int dim, float m, float l) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int i = 0; i < 6; ++i) s.q[i] = lane + 32 * i < dim ? to_f32(q[lane + 32 * i]) : 0.f;
#pragma unroll
    for (int i = 0; i < 4; ++i) s.o[i] = 0.f;
    s.m = m;
    s.l = l;
}
// one key: its first `own` dimensions at k, the others at k_shared; false once every column is NaN for good
template <int MODE>
__device__ __forceinline__ bool plain_key(PlainRow& s, const CachedAttnArgs& a, const __nv_bfloat16* k, int own, const __nv_bfloat16* k_shared,
                                          const __nv_bfloat16* v, int h, int dist) {
    const int lane = threadIdx.x & 31;
    float dot = 0.f;
#pragma unroll
    for (int i = 0; i < 6; ++i) {
        const int d = lane + 32 * i;
        if (d < a.dim) dot = fmaf(s.q[i], to_f32(d < own ? k[d] : k_shared[d - own]), dot);
    }
#pragma unroll
    for (int w = 16; w > 0; w >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, w);
    float p;
    if (MODE == UMBS_ATTN_SIGMOID) {
        p = sigmoidf_(dot * a.scale + (a.head_bias ? a.head_bias[h] : 0.f));
    } else {
        const float sc = shaped_score(a, dot, a.r1 ? a.r1[h] : 0.f, a.r1 ? a.r2[h] : 0.f, dist);
        const float mn = fmaxf(s.m, sc), ref = mn > -INFINITY ? mn : 0.f, corr = expf(s.m - ref);       // (m = -inf: corr = 0)
        p = expf(sc - ref);
        s.l = s.l * corr + p;
        s.m = mn;
#pragma unroll
        for (int i = 0; i < 4; ++i) s.o[i] *= corr;
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
        if (lane + 32 * i < a.vdim) s.o[i] = fmaf(p, to_f32(v[lane + 32 * i]), s.o[i]);
    return MODE == UMBS_ATTN_SIGMOID ? p == p : s.l == s.l;
}

// blocks of `pool` tokens that lie wholly before the window of the row at position p
__device__ __forceinline__ int pooled_visible(int p, int window, int pool) {
    const int lim = p - window + 1;                   // tokens [0, lim) have left the window
    return (pool > 0 && lim >= pool) ? lim / pool : 0;
}

// Keys and values that all sit in the step (seq_window_attn.cu): a head's own key part, a part all heads share, its values.
struct StepKeys {
    const void* q; int64_t ldq;
    const void* k; int64_t ldk; int kdim;
    const void* ks; int64_t ldks;
    const void* v; int64_t ldv;
    void* out; int64_t ldo;
};

// seq_attn_tc.cu, bf16 storage: true if the kernel takes these sizes, strides and addresses.  keys NULL: the step's rows,
// cache and blocks of `a`; else `a` gives sizes (dim: own and shared part together), mask, sink and gate.
bool attention_tc_fits(const CachedAttnArgs& a, const StepKeys* keys);
int launch_attention_tc(int mode, const CachedAttnArgs& a, const StepKeys* keys, const Batch& b, cudaStream_t st);

}  // namespace umbs
