// Matrix memories with one decay per head (seq_chunk.h, retention) on the 5th-generation tensor cores: a prompt's tokens 128 at a time,
// every 128 of them in blocks of their own.  With D[i][j] = decay^(i - j) for j <= i, else 0, and S the state in front of the 128:
//     states   L = (diag(decay^(n - 1 - j)) K)^T V                      a block per 128 tokens, head and 128 value columns
//     chain    S <- decay^n S + L, from the slot's state to the slot's state, every S kept: a thread per element
//     outputs  O = diag(decay^(i + 1)) Q S + ((Q K^T) o D) V            a block as for the states; then the head's norm and gate
// Every operand is 32-bit and taken as three bf16 parts in six products (seq_gemm_split.cu); a product's leading part is summed over at
// most 128 of k and apart from the small ones, so no chain through the tensor core is longer than eight.  Sums whose parts are no
// numbers (operands infinite, NaN or beyond 2^103; sums beyond 2^79) are worked out again in plain fp32.
//
// Bound: what a block does one after the other (rows in, split, products, weights split again, products, out), four warps a scheduler
// in step: outputs 33,000 clocks a block, of which the products take 6,000, three and a half blocks to an SM (192 KB of shared memory
// and all of tensor memory each); states three blocks to an SM (72 KB).  4096 tokens of 16 heads 64 x 128: 238 us in pieces of 32
// tokens on the multiply-add pipe with a norm-and-gate kernel behind, 119 here (states 31, chain 9, outputs 77, cold).  Distance from
// float64 2.1e-7 -> 1.1e-7 (fp32 results of 128 to 1500 tokens), states 1.7e-7 -> 0.9e-7.
#include <math.h>

#include "seq_chunk.h"
#include "seq_tc.cuh"

namespace umbs {

constexpr int kCtT = 128, kCtStride = 132;                  // tokens of a block; floats between rows of results
constexpr int kCtStates = 1024 + 3 * (64 * 128 * 2 + 64 * 128);             // V and K of 64 tokens
constexpr int kCtOutputs = 1024 + 3 * (128 * 128 + 128 * 128 + 128 * 256);  // Q, K (then the state), V

__device__ __forceinline__ void ld8(const float* p, float (&f)[8]) {
    const float4 a = *reinterpret_cast<const float4*>(p), b = *reinterpret_cast<const float4*>(p + 4);
    f[0] = a.x; f[1] = a.y; f[2] = a.z; f[3] = a.w;
    f[4] = b.x; f[5] = b.y; f[6] = b.z; f[7] = b.w;
}
// Numbers d .. d + 7 of a token's query or key row, scaled and turned (d, dim, half of rot_dims: multiples of 8; zeros behind dim).
__device__ __forceinline__ void turned8(const ChunkMemory& x, int64_t tok, int off, float scale, int d, float (&f)[8]) {
    if (d >= x.dim) {
#pragma unroll
        for (int e = 0; e < 8; ++e) f[e] = 0.f;
        return;
    }
    const float* row = x.x + tok * x.ld + off;
    ld8(row + d, f);
#pragma unroll
    for (int e = 0; e < 8; ++e) f[e] *= scale;
    if (d >= x.rot_dims) return;
    const int half = x.rot_dims / 2;
    const bool low = d < half;
    const float* tab = x.rot_tab + tok * x.rot_dims + (low ? d : d - half);
    float g[8], c[8], s[8];
    ld8(row + (low ? d + half : d - half), g);
    ld8(tab, c);
    ld8(tab + half, s);
#pragma unroll
    for (int e = 0; e < 8; ++e) f[e] = low ? f[e] * c[e] - g[e] * scale * s[e] : f[e] * c[e] + g[e] * scale * s[e];
}
// The same for numbers 8 ch .. 8 ch + 7 of a row whose pieces the eight lanes of a row hold in f, with the turn's cos and sin.
__device__ __forceinline__ void load_turn(const ChunkMemory& x, int64_t tok, int ch, float (&c)[8], float (&s)[8]) {
    const int hc = x.rot_dims / 16;
    if (ch >= 2 * hc) return;
    const float* tab = x.rot_tab + tok * x.rot_dims + (ch < hc ? ch : ch - hc) * 8;
    ld8(tab, c);
    ld8(tab + x.rot_dims / 2, s);
}
__device__ __forceinline__ void turn_row(const ChunkMemory& x, int ch, float (&f)[8], const float (&c)[8], const float (&s)[8]) {
    const int hc = x.rot_dims / 16, lane = threadIdx.x & 31;
    const int from = (lane & ~7) | (ch < hc ? ch + hc : (ch < 2 * hc ? ch - hc : ch));
#pragma unroll
    for (int e = 0; e < 8; ++e) {
        const float g = __shfl_sync(0xffffffffu, f[e], from);
        if (ch < 2 * hc) f[e] = ch < hc ? f[e] * c[e] - g * s[e] : f[e] * c[e] + g * s[e];
    }
}
template <bool SCALED = false>
__device__ __forceinline__ void st_parts(uint32_t at, uint32_t step, const float (&f)[8]) {
    uint4 v[3];
    split8<SCALED>(f, v);
#pragma unroll
    for (int e = 0; e < 3; ++e)
        asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(at + e * step), "r"(v[e].x), "r"(v[e].y), "r"(v[e].z), "r"(v[e].w) : "memory");
}
__device__ __forceinline__ bool no_number(float v) { return !(fabsf(v) <= 3.402823466e38f); }
// an operand whose k runs down the rows: its 64-wide pieces are `piece` bytes apart, groups of eight rows 1024
__device__ __forceinline__ uint64_t mn_desc(uint32_t addr, uint32_t piece) {
    return (umb::umma_smem_desc_sw128(addr) & ~((uint64_t)0x3fff << 16)) | ((uint64_t)(piece >> 4) << 16);
}

// What the parts do not give, in plain fp32, by the whole block where one of its sums is no number (prompts of 4096 tokens, 16 heads, all of them
// NaN from the first tokens on: 0.8 ms; each number by a thread of its own, token by token, took 2400 of them).
// The turned and scaled rows of the block's tokens, to rows of dim + 1 floats.
__device__ __forceinline__ void plain_rows(const ChunkMemory& x, int64_t tok, int nb, int off, float scale, float* to) {
    const int n8 = x.dim / 8;
    for (int e = threadIdx.x; e < nb * n8; e += blockDim.x) {
        const int r = e / n8, d = (e - r * n8) * 8;
        float f[8];
        turned8(x, tok + r, off, scale, d, f);
#pragma unroll
        for (int u = 0; u < 8; ++u) to[r * (x.dim + 1) + d + u] = f[u];
    }
}
// L, token by token: dimensions d0 + i of column c for the bits i of odd, to `out` and x.vdim further each
__device__ __noinline__ void plain_states(const ChunkMemory& x, int64_t tok, int nb, int h, int d0, int c, float dec, float* sm, uint32_t odd, float* out) {
    plain_rows(x, tok, nb, x.koff + h * x.dim, x.kscale, sm);
    __syncthreads();
    if (odd == 0) return;
    float s[32] = {};
    const float* v = x.x + tok * x.ld + x.voff + h * x.vdim + c;
    for (int j = 0; j < nb; ++j, v += x.ld) {
        const float z = *v;
#pragma unroll
        for (int i = 0; i < 32; ++i)
            if (odd >> i & 1) s[i] = fmaf(s[i], dec, sm[j * (x.dim + 1) + d0 + i] * z);
    }
#pragma unroll
    for (int i = 0; i < 32; ++i)
        if (odd >> i & 1) out[(int64_t)i * x.vdim] = s[i];
}
// O: columns c + e of row i for the bits e of odd, of `cols` that there are; st: the state in front of the tokens
__device__ __noinline__ void plain_outputs(const ChunkMemory& x, int64_t tok, int nb, int h, int i, int c, int cols, const float* lam, const float* st, float* sm,
                                           uint32_t odd, float* o) {
    const int dp = x.dim + 1;
    float *q = sm, *k = q + kCtT * dp, *w = k + kCtT * dp;  // rows of q and k, weights in rows of kCtT + 1
    plain_rows(x, tok, nb, x.qoff + h * x.dim, x.qscale, q);
    plain_rows(x, tok, nb, x.koff + h * x.dim, x.kscale, k);
    __syncthreads();
    for (int e = threadIdx.x; e < nb * nb; e += blockDim.x) {
        const int r = e / nb, j = e - r * nb;
        if (j > r) continue;
        float z = 0.f;
        for (int d = 0; d < x.dim; ++d) z = fmaf(q[r * dp + d], k[j * dp + d], z);
        w[r * (kCtT + 1) + j] = z * lam[r - j];
    }
    __syncthreads();
    if (odd == 0) return;
    float s[32] = {};
    auto add = [&](float z, const float* row) {
#pragma unroll
        for (int e = 0; e < 32; e += 4)
            if (e < cols) {
                const float4 v = *reinterpret_cast<const float4*>(row + e);
                s[e] = fmaf(z, v.x, s[e]);
                s[e + 1] = fmaf(z, v.y, s[e + 1]);
                s[e + 2] = fmaf(z, v.z, s[e + 2]);
                s[e + 3] = fmaf(z, v.w, s[e + 3]);
            }
    };
    for (int d = 0; d < x.dim; ++d) add(q[i * dp + d], st + (int64_t)d * x.vdim + c);
#pragma unroll
    for (int e = 0; e < 32; ++e) s[e] *= lam[i + 1];
    const float* v = x.x + tok * x.ld + x.voff + h * x.vdim + c;
    for (int j = 0; j <= i; ++j, v += x.ld) add(w[i * (kCtT + 1) + j], v);
#pragma unroll
    for (int e = 0; e < 32; ++e) o[e] = odd >> e & 1 ? s[e] : o[e];
}

__global__ void __launch_bounds__(256, 3) chunk_states_kernel(const __grid_constant__ ChunkMemory x, const __grid_constant__ Batch b, unsigned int* report) {
    extern __shared__ unsigned char smem_raw[];
    __shared__ uint64_t done;
    __shared__ uint32_t s_tmem;
    __shared__ int s_quit, s_odd;
    __shared__ float keep[kCtT];
    volatile int* quit = &s_quit;
    unsigned char* smem = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    chain_wait_only();
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    const int s = blockIdx.x / x.n_seg, c = blockIdx.x - s * x.n_seg, h = blockIdx.y, c0 = blockIdx.z * 128;
    const int t0 = c * kCtT, nb = min(kCtT, b.seq_len[s] - t0);
    const int64_t tok = b.seq_start[s] + t0;
    const float dec = x.decay[h];
    if (nb <= 0) return;
    const int nv = min(128, x.vdim - c0);
    if (tid < kCtT) keep[tid] = tid < nb ? powf(dec, (float)(nb - 1 - tid)) : 0.f;
    if (tid == 0) {
        umb::mbar_init(&done, 1);
        s_quit = s_odd = 0;
        umb::fence_barrier_init();
    }
    if (warp == 0) {
        umb::tmem_alloc(&s_tmem, 128);
        umb::tmem_relinquish();
        chain_next();
    }
    umb::tc_fence_before();
    __syncthreads();
    umb::tc_fence_after();
    const uint32_t tmem = s_tmem, s_v = smem_u32(smem), s_k = s_v + 3 * 16384;
    constexpr uint32_t idesc = tc_idesc(128, 64, true) | (1u << 15);
    bool ok = true;
    for (int half = 0; half < 2 && half * 64 < nb && ok; ++half) {
        const int ch = tid & 7, r8 = tid >> 3, cv = tid & 15, r16 = tid >> 4;
        float kf[2][8] = {}, cf[2][8], sf[2][8];            // asked for ahead of the wait
#pragma unroll
        for (int p = 0; p < 2; ++p) {
            const int j = half * 64 + r8 + 32 * p;
            if (j < nb && ch * 8 < x.dim) {
                ld8(x.x + (tok + j) * x.ld + x.koff + h * x.dim + ch * 8, kf[p]);
                load_turn(x, tok + j, ch, cf[p], sf[p]);
            }
        }
        if (half == 1 && !(ok = __syncthreads_and(tc_spin_warp(&done, 0, quit)))) break;
#pragma unroll
        for (int p = 0; p < 2; ++p) {
            const int r = r8 + 32 * p;
            turn_row(x, ch, kf[p], cf[p], sf[p]);
            const float w = keep[half * 64 + r];
#pragma unroll
            for (int e = 0; e < 8; ++e) kf[p][e] = w == 0.f ? 0.f : kf[p][e] * (x.kscale * kSplitScale) * w;     // (tokens that are not there, or forgotten: nothing)
            st_parts<true>(s_k + r * 128 + ((ch ^ (r & 7)) << 4), 8192, kf[p]);
        }
#pragma unroll
        for (int p = 0; p < 4; ++p) {
            const int r = r16 + 16 * p;
            float f[8] = {};
            if (half * 64 + r < nb && cv * 8 < nv) ld8(x.x + (tok + half * 64 + r) * x.ld + x.voff + h * x.vdim + c0 + cv * 8, f);
            // (the loads stay apart from the multiplications, which the compiler otherwise waits for load by load: 29.8 -> 25.7 us)
            asm volatile("" : "+f"(f[0]), "+f"(f[1]), "+f"(f[2]), "+f"(f[3]), "+f"(f[4]), "+f"(f[5]), "+f"(f[6]), "+f"(f[7]));
            st_parts(s_v + (cv >> 3) * 8192 + r * 128 + (((cv & 7) ^ (r & 7)) << 4), 16384, f);
        }
        umb::fence_proxy_async_smem();
        __syncthreads();
        if (warp == 0) {
            const uint64_t vd = mn_desc(s_v, 8192), kd = mn_desc(s_k, 8192);
            const uint32_t more = half ? 1u : 0u;
            if (umb::elect_one()) {
#pragma unroll
                for (int i = 0; i < 3; ++i)
#pragma unroll
                    for (int j = 0; j < 3 - i; ++j)
#pragma unroll
                        for (int kk = 0; kk < 4; ++kk)
                            umb::umma_ss_f16(tmem + (i + j ? 64 : 0), vd + i * (16384 >> 4) + kk * (2048 >> 4), kd + j * (8192 >> 4) + kk * (2048 >> 4), idesc,
                                             kk > 0 || i > 0 || j > 1 ? 1u : more);
                umb::umma_commit(&done);
            }
            __syncwarp();
        }
    }
    if (ok) ok = __syncthreads_and(tc_spin_warp(&done, nb > 64 ? 1 : 0, quit));
    // lane: value column; 32 dimensions a warp
    const int q = warp & 3, d0 = (warp >> 2) * 32, col = q * 32 + lane;
    float* out = x.seg_state + ((((int64_t)s * x.n_seg + c) * x.heads + h) * x.dim + d0) * x.vdim + c0 + col;
    uint32_t odd = 0;
    if (ok) {
        umb::tc_fence_after();
        const uint32_t at = tmem + ((uint32_t)(q * 32) << 16) + d0;
        uint32_t u[32], v[32];
        UMB_TMEM_LD_X32(at, u);
        UMB_TMEM_LD_X32(at + 64, v);
        umb::tc_wait_ld();
        if (col < nv)
#pragma unroll
            for (int i = 0; i < 32; ++i)
                if (d0 + i < x.dim) {
                    const float l = (__uint_as_float(u[i]) + __uint_as_float(v[i])) * kSplitBack;
                    odd |= (uint32_t)no_number(l) << i;
                    out[(int64_t)i * x.vdim] = l;
                }
        if (odd) s_odd = 1;
    }
    __syncwarp();
    umb::tc_fence_before();
    __syncthreads();
    if (s_odd) plain_states(x, tok, nb, h, d0, min(c0 + col, x.vdim - 1), dec, reinterpret_cast<float*>(smem), odd, out);
    tc_settle(quit, report);
    if (warp == 0) {
        umb::tc_fence_after();
        umb::tmem_dealloc(tmem, 128);
    }
}

// A thread per state element: every L is replaced by the state in front of its tokens; eight of them are on their way at a time.
__global__ void chunk_chain_kernel(const ChunkMemory x, const Batch b) {
    chain_wait();
    const int64_t plane = (int64_t)x.heads * x.dim * x.vdim, e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int s = blockIdx.y, len = b.seq_len[s];
    if (e >= plane || len <= 0) return;
    const int n = (len + kCtT - 1) / kCtT;
    const float dec = x.decay[(int)e / (x.dim * x.vdim)], whole = powf(dec, (float)kCtT), rest = powf(dec, (float)(len - (n - 1) * kCtT));
    float* slot = x.state + (int64_t)b.seq_slot[s] * plane + e;
    float* p = x.seg_state + (int64_t)s * x.n_seg * plane + e;
    float S = b.seq_pos0[s] > 0 ? *slot : 0.f, l[8];
    auto fetch = [&](int c) {
#pragma unroll
        for (int i = 0; i < 8; ++i) l[i] = c + i < n ? p[(c + i) * plane] : 0.f;
    };
    fetch(0);
    for (int c = 0; c < n; c += 8) {
        float f[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) f[i] = l[i];
        if (c + 8 < n) fetch(c + 8);
#pragma unroll
        for (int i = 0; i < 8; ++i)
            if (c + i < n) {
                p[(c + i) * plane] = S;
                S = fmaf(c + i + 1 < n ? whole : rest, S, f[i]);
            }
    }
    *slot = S;
}

// T: the result's type; float with NORM false: o as it is, for a norm over several heads
template <typename T, bool NORM>
__global__ void __launch_bounds__(512, 1) chunk_outputs_kernel(const __grid_constant__ ChunkMemory x, const __grid_constant__ Batch b, float eps, T* __restrict__ out,
                                                               unsigned int* report) {
    extern __shared__ unsigned char smem_raw[];
    __shared__ uint64_t done;
    __shared__ uint32_t s_tmem;
    __shared__ int s_quit, s_bad, s_odd;
    __shared__ float lam[kCtT + 1];
    volatile int* quit = &s_quit;
    unsigned char* smem = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    chain_wait_only();
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    const int s = blockIdx.x / x.n_seg, c = blockIdx.x - s * x.n_seg, h = blockIdx.y, c0 = blockIdx.z * 128;
    const int t0 = c * kCtT, nb = min(kCtT, b.seq_len[s] - t0);
    const int64_t tok = b.seq_start[s] + t0;
    const float dec = x.decay[h];
    if (nb <= 0) return;
    const int nv = min(128, x.vdim - c0);
    if (tid <= kCtT) lam[tid] = powf(dec, (float)tid);
    if (tid == 0) {
        umb::mbar_init(&done, 1);
        s_quit = s_odd = 0;
        s_bad = kCtT;
        umb::fence_barrier_init();
    }
    if (warp == 0) {
        umb::tmem_alloc(&s_tmem, 512);
        umb::tmem_relinquish();
        chain_next();
    }
    const uint32_t s_q = smem_u32(smem), s_k = s_q + 3 * 16384, s_v = s_k + 3 * 16384;
    const int ch = tid & 7, r8 = tid >> 3, cv = tid & 15, r16 = tid >> 4;
    {
        float qf[2][8] = {}, kf[2][8] = {}, cf[2][8], sf[2][8];
#pragma unroll
        for (int p = 0; p < 2; ++p) {
            const int r = r8 + 64 * p;
            if (r < nb && ch * 8 < x.dim) {
                const float* row = x.x + (tok + r) * x.ld + h * x.dim + ch * 8;
                ld8(row + x.qoff, qf[p]);
                ld8(row + x.koff, kf[p]);
                load_turn(x, tok + r, ch, cf[p], sf[p]);
            }
        }
#pragma unroll
        for (int p = 0; p < 2; ++p) {
            const int r = r8 + 64 * p;
            const uint32_t at = r * 128 + ((ch ^ (r & 7)) << 4);
            turn_row(x, ch, qf[p], cf[p], sf[p]);
            turn_row(x, ch, kf[p], cf[p], sf[p]);
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                qf[p][e] *= x.qscale * kSplitScale;
                kf[p][e] *= x.kscale * kSplitScale;
            }
            st_parts<true>(s_q + at, 16384, qf[p]);
            st_parts<true>(s_k + at, 16384, kf[p]);
        }
    }
    // values and state, while the scores are worked out
    const float* st = x.seg_state + (((int64_t)s * x.n_seg + c) * x.heads + h) * x.dim * x.vdim;
    float vf[4][8] = {}, sf[2][8] = {};
#pragma unroll
    for (int p = 0; p < 4; ++p) {
        const int r = r16 + 32 * p;
        if (r < nb && cv * 8 < nv) ld8(x.x + (tok + r) * x.ld + x.voff + h * x.vdim + c0 + cv * 8, vf[p]);
    }
#pragma unroll
    for (int p = 0; p < 2; ++p) {
        const int d = r16 + 32 * p;
        if (d < x.dim && cv * 8 < nv) ld8(st + (int64_t)d * x.vdim + c0 + cv * 8, sf[p]);
    }
    umb::fence_proxy_async_smem();
    umb::tc_fence_before();
    __syncthreads();
    umb::tc_fence_after();
    // tensor memory: scores 0-127 and their small terms 128-255, later the weights' parts 0-63, 64-127, 128-191; results 256-383, 384-511
    const uint32_t tmem = s_tmem;
    if (warp == 0) {
        const uint64_t qd = umb::umma_smem_desc_sw128(s_q), kd = umb::umma_smem_desc_sw128(s_k);
        if (umb::elect_one()) {
#pragma unroll
            for (int i = 0; i < 3; ++i)
#pragma unroll
                for (int j = 0; j < 3 - i; ++j)
#pragma unroll
                    for (int kk = 0; kk < 4; ++kk)
                        umb::umma_ss_f16(tmem + (i + j ? 128 : 0), qd + i * (16384 >> 4) + kk * 2, kd + j * (16384 >> 4) + kk * 2, tc_idesc(128, 128),
                                         kk > 0 || i > 0 || j > 1 ? 1u : 0u);
            umb::umma_commit(&done);
        }
        __syncwarp();
    }
#pragma unroll
    for (int p = 0; p < 4; ++p) {
        const int r = r16 + 32 * p;
        // a weight of 0 times a value that is no number is none either: such values stay out of the product, and the rows from their token
        // on are worked out in plain fp32 (the rows in front of it keep their bits)
        bool bad = false;
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            const bool no = !(fabsf(vf[p][e]) <= 0x1.fep103f);
            bad |= no;
            vf[p][e] = no ? 0.f : vf[p][e];
        }
        if (bad) atomicMin(&s_bad, r);
        st_parts(s_v + (cv >> 3) * 16384 + r * 128 + (((cv & 7) ^ (r & 7)) << 4), 32768, vf[p]);
    }
    // row i: the row of this thread, of which it has 32 columns
    const int q = warp & 3, part = (warp >> 2) * 32, i = q * 32 + lane;
    const uint32_t row = tmem + ((uint32_t)(q * 32) << 16);
    float o[32];
    bool ok = __syncthreads_and(tc_spin_warp(&done, 0, quit));
    if (ok) {
        umb::tc_fence_after();
        uint32_t u[32], v[32];
        UMB_TMEM_LD_X32(row + part, u);
        UMB_TMEM_LD_X32(row + 128 + part, v);
        umb::tc_wait_ld();
#pragma unroll
        for (int p = 0; p < 2; ++p) {                       // the keys have been read: the state takes their place
            const int d = r16 + 32 * p;
            st_parts(s_k + (cv >> 3) * 8192 + d * 128 + (((cv & 7) ^ (d & 7)) << 4), 16384, sf[p]);
        }
        umb::fence_proxy_async_smem();
        umb::tc_fence_before();
        __syncthreads();                                    // (and every thread has read its scores)
        if (warp == 0) {
            umb::tc_fence_after();
            const uint64_t qd = umb::umma_smem_desc_sw128(s_q), sd = mn_desc(s_k, 8192);
            if (umb::elect_one()) {
#pragma unroll
                for (int a = 0; a < 3; ++a)
#pragma unroll
                    for (int j = 0; j < 3 - a; ++j)
#pragma unroll
                        for (int kk = 0; kk < 4; ++kk)
                            umb::umma_ss_f16(tmem + (a + j ? 384 : 256), qd + a * (16384 >> 4) + kk * 2, sd + j * (16384 >> 4) + kk * (2048 >> 4),
                                             tc_idesc(128, 128, true), kk > 0 || a > 0 || j > 1 ? 1u : 0u);
                umb::umma_commit(&done);
            }
            __syncwarp();
        }
        uint32_t w0[16], w1[16], w2[16];                    // weights of two tokens each, in three parts
#pragma unroll
        for (int e = 0; e < 16; ++e) {
            float p[2];
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                const int far = i - (part + 2 * e + k);
                const float z = (__uint_as_float(u[2 * e + k]) + __uint_as_float(v[2 * e + k])) * (kSplitBack * kSplitScale);    // (as split8: 2^24)
                p[k] = far >= 0 ? z * lam[far >= 0 ? far : 0] : 0.f;        // (chosen: a later token's NaN stays its own)
            }
            uint32_t* to[3] = {&w0[e], &w1[e], &w2[e]};
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                const __nv_bfloat162 r = __floats2bfloat162_rn(p[0], p[1]);
                const uint32_t bits = *reinterpret_cast<const uint32_t*>(&r);
                *to[k] = bits;
                p[0] -= __uint_as_float(bits << 16);
                p[1] -= __uint_as_float(bits & 0xffff0000u);
            }
        }
        UMB_TMEM_ST_X16(row + part / 2, w0);
        UMB_TMEM_ST_X16(row + 64 + part / 2, w1);
        UMB_TMEM_ST_X16(row + 128 + part / 2, w2);
        umb::tc_wait_st();
        ok = __syncthreads_and(tc_spin_warp(&done, 1, quit));
    }
    if (ok) {
        umb::tc_fence_after();
        uint32_t u[32], v[32];
        UMB_TMEM_LD_X32(row + 256 + part, u);
        UMB_TMEM_LD_X32(row + 384 + part, v);
        umb::tc_wait_ld();
        const float f = lam[i + 1];
#pragma unroll
        for (int e = 0; e < 32; ++e) o[e] = f * ((__uint_as_float(u[e]) + __uint_as_float(v[e])) * kSplitBack);
        umb::tc_fence_before();
        __syncthreads();
        if (warp == 0) {
            umb::tc_fence_after();
            const uint64_t vd = mn_desc(s_v, 16384);
            if (umb::elect_one()) {
#pragma unroll
                for (int a = 0; a < 3; ++a)
#pragma unroll
                    for (int j = 0; j < 3 - a; ++j)
#pragma unroll
                        for (int kk = 0; kk < 8; ++kk)
                            umb::umma_ts_f16(tmem + (a + j ? 384 : 256), tmem + a * 64 + kk * 8, vd + j * (32768 >> 4) + kk * (2048 >> 4), tc_idesc(128, 128, true),
                                             kk > 0 || a > 0 || j > 1 ? 1u : 0u);
                umb::umma_commit(&done);
            }
            __syncwarp();
        }
        ok = __syncthreads_and(tc_spin_warp(&done, 0, quit));
    }
    if (ok) {
        umb::tc_fence_after();
        uint32_t u[32], v[32];
        UMB_TMEM_LD_X32(row + 256 + part, u);
        UMB_TMEM_LD_X32(row + 384 + part, v);
        umb::tc_wait_ld();
        const int n0 = c0 + part;                           // this thread's first column
        uint32_t odd = 0;
#pragma unroll
        for (int e = 0; e < 32; ++e) {
            o[e] += (__uint_as_float(u[e]) + __uint_as_float(v[e])) * kSplitBack;
            odd |= (uint32_t)((i >= s_bad || no_number(o[e])) && i < nb) << e;
        }
        if (odd) s_odd = 1;
        // rows leave by whole warps, four columns a lane, from where the values were (a thread's own row, 16 bytes of it at a time beside 31
        // others, took 15,000 clocks of 35,000)
        float* so = reinterpret_cast<float*>(smem + 6 * 16384);
        auto put = [&] {
#pragma unroll
            for (int e = 0; e < 32; e += 4) *reinterpret_cast<float4*>(so + i * kCtStride + part + e) = make_float4(o[e], o[e + 1], o[e + 2], o[e + 3]);
            __syncthreads();
        };
        put();
        if (s_odd) {
            float f[32];                                    // (columns that are not there: 0 times a score beyond the parts is none)
#pragma unroll
            for (int e = 0; e < 32; ++e) {
                f[e] = part + e < nv ? o[e] : 0.f;
                odd &= ~((uint32_t)(part + e >= nv) << e);
            }
            plain_outputs(x, tok, nb, h, i, n0, nv - part, lam, st, reinterpret_cast<float*>(smem), odd, f);
#pragma unroll
            for (int e = 0; e < 32; ++e) o[e] = f[e];
            __syncthreads();
            put();
        }
        const int hv = x.heads * x.vdim, rows = min(8, nb - warp * 8);
        const float* g = x.x + (tok + warp * 8) * x.ld + x.voff + hv + (int64_t)h * x.vdim + c0 + lane * 4;
        T* orow = out + (tok + warp * 8) * hv + (int64_t)h * x.vdim + c0 + lane * 4;
        float4 gv[8];
        if (NORM && lane * 4 < nv)
#pragma unroll
            for (int r = 0; r < 8; ++r)
                if (r < rows) gv[r] = *reinterpret_cast<const float4*>(g + r * x.ld);
        float4 f[8];
        float inv = 1.f;
#pragma unroll
        for (int r = 0; r < 8; ++r)                         // (columns that are not there: 0, and NaN beside a score beyond the parts)
            f[r] = lane * 4 < nv ? *reinterpret_cast<const float4*>(so + (warp * 8 + r) * kCtStride + lane * 4) : make_float4(0.f, 0.f, 0.f, 0.f);
        if (NORM) {                                         // o / rms(o) over the head, times silu(g): lane r has row r's factor
            float ss = 0.f;
#pragma unroll
            for (int r = 0; r < 8; ++r) {
                float z = fmaf(f[r].x, f[r].x, fmaf(f[r].y, f[r].y, fmaf(f[r].z, f[r].z, f[r].w * f[r].w)));
#pragma unroll
                for (int w = 16; w > 0; w >>= 1) z += __shfl_xor_sync(0xffffffffu, z, w);
                if (lane == r) ss = z;
            }
            inv = 1.f / sqrtf(ss / (float)x.vdim + eps);
        }
#pragma unroll
        for (int r = 0; r < 8; ++r) {
            if (r >= rows) continue;
            float z[4] = {f[r].x, f[r].y, f[r].z, f[r].w};
            if (NORM) {
                const float by = __shfl_sync(0xffffffffu, inv, r), ga[4] = {gv[r].x, gv[r].y, gv[r].z, gv[r].w};
#pragma unroll
                for (int k = 0; k < 4; ++k) z[k] = z[k] * by * (ga[k] / (1.f + expf(-ga[k])));         // (retention_gate_kernel's)
            }
            if (lane * 4 >= nv) continue;
            T* to = orow + (int64_t)r * hv;
            if constexpr (sizeof(T) == 4) {
                *reinterpret_cast<float4*>(to) = make_float4(z[0], z[1], z[2], z[3]);
            } else {
                const __nv_bfloat162 a = __floats2bfloat162_rn(z[0], z[1]), d = __floats2bfloat162_rn(z[2], z[3]);
                *reinterpret_cast<uint2*>(to) = make_uint2(*reinterpret_cast<const uint32_t*>(&a), *reinterpret_cast<const uint32_t*>(&d));
            }
        }
    }
    __syncwarp();
    umb::tc_fence_before();
    __syncthreads();
    tc_settle(quit, report);
    if (warp == 0) {
        umb::tc_fence_after();
        umb::tmem_dealloc(tmem, 512);
    }
}

int chunk_tc_count(const ChunkMemory& m, const Batch& b, const void* out, size_t fit) {
    const int n = (b.max_seq_len + kCtT - 1) / kCtT;
    auto al = [](const void* p) { return ((uintptr_t)p & 15) == 0; };
    if (m.gates != nullptr || m.normaliser || m.dim % 8 || m.dim > 64 || m.vdim % 8 || m.rot_dims % 16 || b.max_seq_len < kCtT || (size_t)n > fit) return 0;
    if (m.ld % 4 || m.qoff % 4 || m.koff % 4 || m.voff % 4 || !al(m.x) || !al(m.seg_state) || !al(out) || (m.rot_dims > 0 && !al(m.rot_tab))) return 0;
    return n;
}

template <typename T, bool NORM>
static int launch_outputs(const ChunkMemory& m, const Batch& b, const dim3& grid, float eps, T* out, unsigned int* report, cudaStream_t st) {
    auto kernel = chunk_outputs_kernel<T, NORM>;
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kCtOutputs);
    return e != cudaSuccess ? (int)e : chain_launch(kernel, grid, 512, kCtOutputs, st, m, b, eps, out, report);
}

int launch_chunk_tc(const ChunkMemory& m, const Batch& b, int norm_dtype, float eps, void* out, cudaStream_t st) {
    unsigned int* report = nullptr;
    int rc = give_up_word(&report);
    if (rc == 0) rc = give_up_status();
    if (rc != 0) return rc;
    const dim3 grid(b.n_seqs * m.n_seg, m.heads, (m.vdim + 127) / 128);
    const cudaError_t e = cudaFuncSetAttribute(chunk_states_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kCtStates);
    if (e != cudaSuccess) return (int)e;
    rc = chain_launch(chunk_states_kernel, grid, 256, kCtStates, st, m, b, report);
    if (rc != 0) return rc;
    const int64_t plane = (int64_t)m.heads * m.dim * m.vdim;
    rc = chain_launch(chunk_chain_kernel, dim3((unsigned)((plane + 255) / 256), b.n_seqs), 256, 0, st, m, b);
    if (rc != 0) return rc;
    if (norm_dtype == UMBS_BF16) return launch_outputs<__nv_bfloat16, true>(m, b, grid, eps, (__nv_bfloat16*)out, report, st);
    if (norm_dtype == UMBS_F32) return launch_outputs<float, true>(m, b, grid, eps, (float*)out, report, st);
    return launch_outputs<float, false>(m, b, grid, eps, m.out, report, st);
}

unsigned int chunk_tc_timeouts() { return tc_timeouts(); }

}  // namespace umbs
