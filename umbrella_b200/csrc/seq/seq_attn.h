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
