// Attention of a ragged step over a per-slot key/value cache: sliding window (or everything before the row), optionally
// with one mean key/value per block of older tokens, and three ways from scores to weights (softmax, softmax with a
// sink, sigmoid).  A key is read where it lives: tokens of the step from the step's own rows, older tokens from the
// slot's cache rows (position p at row p mod kv_len), pooled blocks from the slot's block table -- so a prompt in one
// piece, in portions, and token-by-token decoding all walk the same keys in the same order.
//
// Steps with several tokens per sequence, bf16, of the sizes and addresses that seq_attn_tc.cu takes: its kernel.
// Tile kernel (any other such step): one block = 64 consecutive query rows of one (sequence, head); 256 threads as 16 x 16, a thread
// owns 4 rows x 4 keys of the score tile and 4 rows x VC value columns of the output; per tile of 64 keys the scores come
// from transposed fp32 tiles in shared memory, the weights go back through shared memory for the value product.  The key
// tile holds 64 dimensions at a time (larger heads add their scores up over several passes), which keeps two blocks on an
// SM for heads of 128.
// Decode kernels (one token per sequence): cached_attention_decode_group_kernel for bf16 rows of up to 128 numbers and more than a few keys; else one block = (sequence, head, split); a warp takes every 8th key of the block's
// share, lanes striding over the head's dimensions; partial (max, sum, output) triples are merged per block and, with more
// than one split, by a second kernel.
// Score options (umbs_attn_opts_t): a tanh cap, a penalty r1 ln(1 + r2 distance) per head, a chunked mask, several maps per
// head and every query head against every value head.  The grid's head axis then counts "virtual heads"
// (h maps + m) value_heads + c, each an independent softmax row; their normalised outputs can be left in fp32
// (raw_out) for umbs_attention_finish, which mixes heads' weights, subtracts maps, norms and gates.
// Everything is fp32 arithmetic; T is the storage type of q, the key/value rows and the output.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <math.h>
#include <algorithm>
#include <stdint.h>

#include "../attn_rules.h"
#include "seq_attn.h"

namespace umbs {

constexpr int kCaQ = 64, kCaK = 64, kCaS = 68;        // rows and keys per tile; row stride of the [d][row] tiles
constexpr int kCaD = 64;                              // dimensions of a key tile held at a time

template <typename T, int VC, int MODE>
__global__ void __launch_bounds__(256) cached_attention_kernel(CachedAttnArgs a, Batch b) {
    extern __shared__ __align__(16) float sm[];
    constexpr int VW = 16 * VC, VP = VW + 4;
    const int dim = a.dim, vdim = a.vdim;
    float* Qs = sm;                                   // [dim][kCaS]  Qs[d][row]
    float* Ks = Qs + (size_t)dim * kCaS;              // [min(dim, kCaD)][kCaS]  Ks[d][key], kCaD dimensions at a time
    float* Vs = Ks + (size_t)min(dim, kCaD) * kCaS;   // [kCaK][VP]
    float* Ps = Vs + (size_t)kCaK * VP;               // [kCaK][kCaS] Ps[key][row]
    const int s = blockIdx.z, vh = blockIdx.y, q0 = blockIdx.x * kCaQ;
    const int len = b.seq_len[s], start = b.seq_start[s], pos0 = b.seq_pos0[s], slot = b.seq_slot[s];
    if (q0 >= len) return;
    const VHead vhd = virtual_head(a, vh);
    const int h = vhd.h, row_kv = vhd.row_kv, koff = vhd.koff, voff = vhd.voff;
    const int window = a.window > 0 ? a.window : (1 << 30), chunk = a.chunk;
    const float r1h = a.r1 ? a.r1[h] : 0.f, r2h = a.r1 ? a.r2[h] : 0.f;
    const T* q = (const T*)a.q;
    const T* kv = (const T*)a.kv;
    const T* cache = (const T*)a.kv_cache;
    const T* pooled = (const T*)a.pool_cache;
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    for (int i = tid; i < kCaQ * dim; i += 256) {
        const int r = i / dim, d = i - r * dim;
        Qs[d * kCaS + r] = (q0 + r < len) ? to_f32(q[(int64_t)(start + q0 + r) * vhd.qstride + vhd.qoff + d]) : 0.f;
    }
    float m[4], l[4], o[4][VC];
    const float sk = MODE == UMBS_ATTN_SOFTMAX_SINK ? sink_score(a, h) : -INFINITY;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        m[i] = sk;                                                     // the sink: a key of this score ...
        l[i] = MODE == UMBS_ATTN_SOFTMAX_SINK ? 1.f : 0.f;             // ... that counts in the sum and has no value
#pragma unroll
        for (int c = 0; c < VC; ++c) o[i][c] = 0.f;
    }
    const float hb = (MODE == UMBS_ATTN_SIGMOID && a.head_bias) ? a.head_bias[h] : 0.f;
    const int p_lo = pos0 + q0, p_hi = pos0 + min(len, q0 + kCaQ) - 1;      // positions of the block's first and last row
    const int n_pool = pooled_visible(p_hi, window, a.pool);               // blocks the last row sees
    const int tiles_pool = (n_pool + kCaK - 1) / kCaK;
    const int j_lo = max(max(0, p_lo - window + 1), chunk > 0 ? p_lo / chunk * chunk : 0);
    const int tiles_tok = (p_hi - j_lo) / kCaK + 1;
    for (int tile = 0; tile < tiles_pool + tiles_tok; ++tile) {
        const bool in_pool = tile < tiles_pool;
        const int base = in_pool ? tile * kCaK : j_lo + (tile - tiles_pool) * kCaK;
        const int hi = in_pool ? n_pool - 1 : p_hi;                        // last index of this kind any row sees
        float sc[4][4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int jj = 0; jj < 4; ++jj) sc[i][jj] = 0.f;
        for (int d0 = 0; d0 < dim; d0 += kCaD) {
            const int dc = min(kCaD, dim - d0);
            __syncthreads();                          // the previous pass or tile is consumed (the very first time: Qs is written)
            for (int i = tid; i < kCaK * dc; i += 256) {
                const int kk = i / dc, d = i - kk * dc, j = base + kk;
                float val = 0.f;
                if (j <= hi) {
                    const T* src = in_pool ? pooled + ((int64_t)slot * a.pool_len + j) * row_kv
                                 : (j >= pos0 ? kv + (int64_t)(start + j - pos0) * row_kv
                                              : cache + ((int64_t)slot * a.kv_len + j % a.kv_len) * row_kv);
                    val = to_f32(src[koff + d0 + d]);
                }
                Ks[d * kCaS + kk] = val;
            }
            for (int i = tid; d0 == 0 && i < kCaK * VW; i += 256) {
                const int kk = i / VW, c = i - kk * VW, j = base + kk;
                float val = 0.f;
                if (j <= hi && c < vdim) {
                    const T* src = in_pool ? pooled + ((int64_t)slot * a.pool_len + j) * row_kv
                                 : (j >= pos0 ? kv + (int64_t)(start + j - pos0) * row_kv
                                              : cache + ((int64_t)slot * a.kv_len + j % a.kv_len) * row_kv);
                    val = to_f32(src[voff + c]);
                }
                Vs[kk * VP + c] = val;
            }
            __syncthreads();
            for (int d = 0; d < dc; ++d) {
                const float4 qv = *reinterpret_cast<const float4*>(Qs + (d0 + d) * kCaS + ty * 4);
                const float4 kv4 = *reinterpret_cast<const float4*>(Ks + d * kCaS + tx * 4);
                const float qa[4] = {qv.x, qv.y, qv.z, qv.w}, ka[4] = {kv4.x, kv4.y, kv4.z, kv4.w};
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int jj = 0; jj < 4; ++jj) sc[i][jj] = fmaf(qa[i], ka[jj], sc[i][jj]);
            }
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int r = q0 + ty * 4 + i, rp = pos0 + r;                  // the row's place in the step and its position
            float p[4];
            bool vis[4];
#pragma unroll
            for (int jj = 0; jj < 4; ++jj) {
                const int j = base + tx * 4 + jj;
                vis[jj] = r < len && (in_pool ? j < pooled_visible(rp, window, a.pool)
                                              : (j <= rp && j > rp - window && (chunk <= 0 || j / chunk == rp / chunk)));
            }
            if (MODE == UMBS_ATTN_SIGMOID) {
#pragma unroll
                for (int jj = 0; jj < 4; ++jj) p[jj] = vis[jj] ? sigmoidf_(sc[i][jj] * a.scale + hb) : 0.f;
            } else {
                float val[4], mx = -INFINITY;
#pragma unroll
                for (int jj = 0; jj < 4; ++jj) {
                    val[jj] = vis[jj] ? shaped_score(a, sc[i][jj], r1h, r2h, rp - (base + tx * 4 + jj)) : -INFINITY;
                    mx = fmaxf(mx, val[jj]);
                }
#pragma unroll
                for (int w = 8; w > 0; w >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, w));   // the row's 16 threads
                const float mn = fmaxf(m[i], mx);
                float sum = 0.f, corr = 1.f;
#pragma unroll
                for (int jj = 0; jj < 4; ++jj) p[jj] = 0.f;
                if (mn > -INFINITY) {
                    corr = expf(m[i] - mn);
#pragma unroll
                    for (int jj = 0; jj < 4; ++jj) {
                        p[jj] = vis[jj] ? expf(val[jj] - mn) : 0.f;
                        sum += p[jj];
                    }
                }
#pragma unroll
                for (int w = 8; w > 0; w >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, w);
                l[i] = l[i] * corr + sum;
                m[i] = mn;
#pragma unroll
                for (int c = 0; c < VC; ++c) o[i][c] *= corr;
            }
#pragma unroll
            for (int jj = 0; jj < 4; ++jj) Ps[(tx * 4 + jj) * kCaS + ty * 4 + i] = p[jj];
        }
        __syncthreads();
        for (int kk = 0; kk < kCaK; ++kk) {
            const float4 pv = *reinterpret_cast<const float4*>(Ps + kk * kCaS + ty * 4);
            const float pa[4] = {pv.x, pv.y, pv.z, pv.w};
#pragma unroll
            for (int cb = 0; cb < VC / 4; ++cb) {
                const float4 vv = *reinterpret_cast<const float4*>(Vs + kk * VP + cb * 64 + tx * 4);
                const float va[4] = {vv.x, vv.y, vv.z, vv.w};
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int c = 0; c < 4; ++c) o[i][cb * 4 + c] = fmaf(pa[i], va[c], o[i][cb * 4 + c]);
            }
        }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int r = q0 + ty * 4 + i;
        if (r >= len) continue;
        const int64_t t = start + r;
        const float inv = MODE == UMBS_ATTN_SIGMOID ? 1.f : 1.f / l[i];
        if (a.raw != nullptr) {
            float* rrow = a.raw + (t * vhd.nv + vh) * vdim;
#pragma unroll
            for (int cb = 0; cb < VC / 4; ++cb)
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    const int col = cb * 64 + tx * 4 + c;
                    if (col < vdim) rrow[col] = o[i][cb * 4 + c] * inv;
                }
            continue;
        }
        const float* grow = a.gate ? a.gate + t * a.ldg + (a.gate_per_head ? h : h * vdim) : nullptr;
        const float gh = (grow && a.gate_per_head) ? sigmoidf_(grow[0]) : 1.f;
        T* orow = (T*)a.out + t * a.heads * vdim + (int64_t)h * vdim;
#pragma unroll
        for (int cb = 0; cb < VC / 4; ++cb)
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const int col = cb * 64 + tx * 4 + c;
                if (col < vdim) {
                    const float gt = (grow && !a.gate_per_head) ? sigmoidf_(grow[col]) : gh;
                    orow[col] = from_f32<T>(o[i][cb * 4 + c] * inv * gt);
                }
            }
    }
}

template <typename T, int VC, int MODE>
static int launch_tiles(const CachedAttnArgs& a, const Batch& b, cudaStream_t st) {
    const size_t smem = ((size_t)(a.dim + std::min(a.dim, kCaD)) * kCaS + (size_t)kCaK * (16 * VC + 4) + (size_t)kCaK * kCaS) * sizeof(float);
    static size_t set = 0;
    if (smem > 48 * 1024 && smem > set) {
        cudaError_t e = cudaFuncSetAttribute(cached_attention_kernel<T, VC, MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)smem);
        if (e != cudaSuccess) return (int)e;
        set = smem;
    }
    const dim3 grid((b.max_seq_len + kCaQ - 1) / kCaQ, a.heads * a.maps * a.vheads, b.n_seqs);
    cached_attention_kernel<T, VC, MODE><<<grid, 256, smem, st>>>(a, b);
    return 0;
}

template <typename T, int MODE>
static int launch_mode(const CachedAttnArgs& a, const Batch& b, cudaStream_t st) {
    if (a.vdim <= 64) return launch_tiles<T, 4, MODE>(a, b, st);
    if (a.vdim <= 128) return launch_tiles<T, 8, MODE>(a, b, st);
    return launch_tiles<T, 16, MODE>(a, b, st);
}

template <typename T>
static int launch_any(int mode, const CachedAttnArgs& a, const Batch& b, cudaStream_t st) {
    switch (mode) {
        case UMBS_ATTN_SOFTMAX: return launch_mode<T, UMBS_ATTN_SOFTMAX>(a, b, st);
        case UMBS_ATTN_SOFTMAX_SINK: return launch_mode<T, UMBS_ATTN_SOFTMAX_SINK>(a, b, st);
        case UMBS_ATTN_SIGMOID: return launch_mode<T, UMBS_ATTN_SIGMOID>(a, b, st);
    }
    return UMB_ERR_ARG;
}


// ------------------------------------------------------------------------------------------------ decode steps
// One block = (split, head, sequence) of a step with one token per sequence.  The row's keys -- pooled blocks first,
// then the tokens of its window -- are numbered 0 .. n - 1 and cut into n_split equal runs; inside a block warp w takes
// keys w, w + 8, ... of the run, lanes striding over the head's dimensions, with its own running (maximum, sum, output).
// The warps' triples are merged in shared memory; one split writes the output itself, several leave their triples in
// `part` [(token, head), split, vdim + 2] for cached_attention_merge_kernel.
constexpr int kCdWarps = 8, kCdMaxPerLane = 8;        // dim, vdim <= 256

template <typename T, int MODE>
__global__ void __launch_bounds__(32 * kCdWarps) cached_attention_decode_kernel(CachedAttnArgs a, Batch b, int n_split,
                                                                                float* __restrict__ part) {
    __shared__ float sm_o[kCdWarps][32 * kCdMaxPerLane];
    __shared__ float sm_ml[kCdWarps][2];
    chain_wait();
    const int split = blockIdx.x, vh = blockIdx.y, s = blockIdx.z;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int dim = a.dim, vdim = a.vdim;
    const int t = b.seq_start[s], p = b.seq_pos0[s], slot = b.seq_slot[s];
    const VHead vhd = virtual_head(a, vh);
    const int h = vhd.h, row_kv = vhd.row_kv, koff = vhd.koff, voff = vhd.voff;
    const float r1h = a.r1 ? a.r1[h] : 0.f, r2h = a.r1 ? a.r2[h] : 0.f;
    const int window = a.window > 0 ? a.window : (1 << 30);
    const int n_pool = pooled_visible(p, window, a.pool);
    const int j_lo = max(max(0, p - window + 1), a.chunk > 0 ? p / a.chunk * a.chunk : 0);
    const int n_keys = n_pool + (p - j_lo + 1);
    const int per = (n_keys + n_split - 1) / n_split, lo = split * per, hi = min(n_keys, lo + per);
    const T* qrow = (const T*)a.q + (int64_t)t * vhd.qstride + vhd.qoff;
    float qv[kCdMaxPerLane], o[kCdMaxPerLane];
#pragma unroll
    for (int i = 0; i < kCdMaxPerLane; ++i) {
        const int d = lane + 32 * i;
        qv[i] = d < dim ? to_f32(qrow[d]) : 0.f;
        o[i] = 0.f;
    }
    const float hb = (MODE == UMBS_ATTN_SIGMOID && a.head_bias) ? a.head_bias[h] : 0.f;
    float m = -INFINITY, l = 0.f;
    // Four of the warp's keys at a time: their key and value loads are all in flight before the first is needed; the
    // softmax state then takes them one by one, in key order (the same additions as one key at a time).
    constexpr int KU = 4;
    for (int kb = lo + w; kb < hi; kb += kCdWarps * KU) {
        const T* src[KU];
        int dist[KU];
        float dot[KU], vv[KU][kCdMaxPerLane];
#pragma unroll
        for (int u = 0; u < KU; ++u) {
            const int k = min(kb + u * kCdWarps, hi - 1);           // (a place beyond the run reads the last key; unused)
            dist[u] = 0;
            if (k < n_pool) src[u] = (const T*)a.pool_cache + ((int64_t)slot * a.pool_len + k) * row_kv;
            else {
                const int j = j_lo + (k - n_pool);
                dist[u] = p - j;
                src[u] = j >= p ? (const T*)a.kv + (int64_t)t * row_kv
                                : (const T*)a.kv_cache + ((int64_t)slot * a.kv_len + j % a.kv_len) * row_kv;
            }
        }
#pragma unroll
        for (int u = 0; u < KU; ++u) {
            dot[u] = 0.f;
#pragma unroll
            for (int i = 0; i < kCdMaxPerLane; ++i) {
                const int d = lane + 32 * i;
                if (d < dim) dot[u] = fmaf(qv[i], to_f32(src[u][koff + d]), dot[u]);
            }
        }
#pragma unroll
        for (int u = 0; u < KU; ++u)
#pragma unroll
            for (int i = 0; i < kCdMaxPerLane; ++i) {
                const int d = lane + 32 * i;
                vv[u][i] = d < vdim ? to_f32(src[u][voff + d]) : 0.f;
            }
#pragma unroll
        for (int x = 16; x > 0; x >>= 1)
#pragma unroll
            for (int u = 0; u < KU; ++u) dot[u] += __shfl_xor_sync(0xffffffffu, dot[u], x);
#pragma unroll
        for (int u = 0; u < KU; ++u) {
            if (kb + u * kCdWarps >= hi) break;
            float pw;
            if (MODE == UMBS_ATTN_SIGMOID) {
                pw = sigmoidf_(dot[u] * a.scale + hb);
            } else {
                const float sc = shaped_score(a, dot[u], r1h, r2h, dist[u]), mn = fmaxf(m, sc), corr = expf(m - mn);   // m = -inf the first time: corr = 0
                pw = expf(sc - mn);
                l = l * corr + pw;
                m = mn;
#pragma unroll
                for (int i = 0; i < kCdMaxPerLane; ++i) o[i] *= corr;
            }
#pragma unroll
            for (int i = 0; i < kCdMaxPerLane; ++i) o[i] = fmaf(pw, vv[u][i], o[i]);
        }
    }
#pragma unroll
    for (int i = 0; i < kCdMaxPerLane; ++i) sm_o[w][lane + 32 * i] = o[i];
    if (lane == 0) { sm_ml[w][0] = m; sm_ml[w][1] = l; }
    __syncthreads();
    // merge the warps' triples (in warp order); thread c < vdim owns output column c
    const int c = threadIdx.x;
    float M = -INFINITY, L = 0.f, O = 0.f;
    if (MODE == UMBS_ATTN_SIGMOID) {
        if (c < vdim)
            for (int ww = 0; ww < kCdWarps; ++ww) O += sm_o[ww][c];
    } else {
        for (int ww = 0; ww < kCdWarps; ++ww) M = fmaxf(M, sm_ml[ww][0]);
        const float sk = (n_split == 1 && MODE == UMBS_ATTN_SOFTMAX_SINK) ? sink_score(a, h) : -INFINITY;
        M = fmaxf(M, sk);
        for (int ww = 0; ww < kCdWarps; ++ww) {
            const float mw = sm_ml[ww][0], f = mw > -INFINITY ? expf(mw - M) : 0.f;
            L = fmaf(sm_ml[ww][1], f, L);
            if (c < vdim) O = fmaf(sm_o[ww][c], f, O);
        }
        if (n_split == 1 && MODE == UMBS_ATTN_SOFTMAX_SINK) L += expf(sk - M);
    }
    if (n_split > 1) {
        float* pr = part + (((int64_t)t * vhd.nv + vh) * n_split + split) * (vdim + 2);
        if (c < vdim) pr[c] = O;
        if (c == 0) { pr[vdim] = M; pr[vdim + 1] = L; }
        return;
    }
    if (c < vdim) {
        const float inv = MODE == UMBS_ATTN_SIGMOID ? 1.f : 1.f / L;
        if (a.raw != nullptr) { a.raw[((int64_t)t * vhd.nv + vh) * vdim + c] = O * inv; return; }
        float gt = 1.f;
        if (a.gate) gt = sigmoidf_(a.gate[(int64_t)t * a.ldg + (a.gate_per_head ? h : h * vdim + c)]);
        ((T*)a.out)[(int64_t)t * a.heads * vdim + (int64_t)h * vdim + c] = from_f32<T>(O * inv * gt);
    }
}

// Decode steps over bf16 rows: the query heads that share a key/value head together, so that a key and a value are fetched
// once for all of them.  One block = (split, up to eight heads of a key/value head, sequence), four or six (NW) warps that each take every
// fourth or sixth tile of 32 keys of the split, with running (maximum, sum, output) of their own.  A tile's rows come to shared memory
// by 16-byte copies, keys and values as groups of their own, the next tile's while this one is worked on.  Both products are
// 16 x 8 x 16 warp-level tensor-core products with the heads as rows (half of the 16 are empty: the step is bound by its
// bytes, and these take a tenth of the instructions that FMAs would): bf16 products are exact, a product's sums are added up
// by ordinary fp32 additions from one k step and one tile to the next (the tensor core would cut them off), and the fp32
// weights go in as three bf16 numbers that add up to them exactly.  The warps' triples are merged in warp order, splits by
// cached_attention_merge_kernel as before.
// 64 sequences x 1040 keys, 16 heads over 4 of 128 (136 MB): a warp per (head, key) took 407 us, heads together with FMAs 65 us,
// this with four warps 51 us in two splits, 43 in one, with six warps 37 (3.7 TB/s).
constexpr int kCgKeys = 32, kCgHeads = 8;

struct GroupSizes { int ks16, vs16, warp_bytes; };          // 16-byte pieces between key rows and between value rows (odd: no bank conflicts)
__host__ __device__ __forceinline__ GroupSizes group_sizes(int dim, int vdim) {
    GroupSizes z;
    z.ks16 = ((dim + 15) / 16 * 2) | 1;
    z.vs16 = (vdim / 8) | 1;
    z.warp_bytes = kCgKeys * (z.ks16 + z.vs16) * 16;
    return z;
}
__device__ __forceinline__ void ldsm4(uint32_t (&r)[4], unsigned addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldsm4t(uint32_t (&r)[4], unsigned addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
// d += a b with the lower eight rows of a empty
__device__ __forceinline__ void mma_top(float (&d)[4], uint32_t a0, uint32_t a2, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%6,%5,%6}, {%7,%8}, {%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a0), "r"(a2), "r"(0u), "r"(b0), "r"(b1));
}

// A warp's triple of one head in plain fp32: every NW-th tile of the keys [lo, hi) from the warp's own, key after key.
template <int MODE, int NW>
__device__ __forceinline__ void plain_part(const CachedAttnArgs& a, const VHead& v, const __nv_bfloat16* q, int h, const __nv_bfloat16* own, int slot, int p, int n_pool,
                                        int j_lo, int first, int hi, float* s_o, float* s_ml) {
    const int lane = threadIdx.x & 31;
    PlainRow s;
    plain_start(s, q, a.dim, -INFINITY, 0.f);
    bool go = true;
    for (int k0 = first; go && k0 < hi; k0 += NW * kCgKeys)
        for (int k = k0; go && k < min(k0 + kCgKeys, hi); ++k) {
            const int j = j_lo + (k - n_pool);
            const __nv_bfloat16* row = k < n_pool ? (const __nv_bfloat16*)a.pool_cache + ((int64_t)slot * a.pool_len + k) * v.row_kv
                                     : j >= p ? own : (const __nv_bfloat16*)a.kv_cache + ((int64_t)slot * a.kv_len + j % a.kv_len) * v.row_kv;
            go = plain_key<MODE>(s, a, row + v.koff, a.dim, nullptr, row + v.voff, h, k < n_pool ? 0 : p - j);
        }
#pragma unroll
    for (int i = 0; i < 4; ++i)
        if (lane + 32 * i < a.vdim) s_o[lane + 32 * i] = s.o[i];
    if (lane == 0) { s_ml[0] = s.m; s_ml[1] = s.l; }
}

template <int MODE, int NW>
__global__ void __launch_bounds__(32 * NW, NW == 4 ? 3 : 2) cached_attention_decode_group_kernel(const __grid_constant__ CachedAttnArgs a, const __grid_constant__ Batch b,
                                                                                         int n_split, float* __restrict__ part) {
    extern __shared__ __align__(16) unsigned char smem[];
    chain_wait();
    const int dim = a.dim, vdim = a.vdim, G = a.heads / a.kv_heads, chunks = (G + kCgHeads - 1) / kCgHeads;
    const GroupSizes z = group_sizes(dim, vdim);
    const int split = blockIdx.x, s = blockIdx.z, lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int gc = blockIdx.y % chunks, kvh = blockIdx.y / chunks;          // which eight of the group's heads
    const int h0 = kvh * G + gc * kCgHeads, nh = min(kCgHeads, G - gc * kCgHeads);
    const VHead v0 = virtual_head(a, h0);                                   // (one map, one value head: the rule asks for a bf16 result)
    const int t = b.seq_start[s], p = b.seq_pos0[s], slot = b.seq_slot[s];
    const int window = a.window > 0 ? a.window : (1 << 30);
    const int n_pool = pooled_visible(p, window, a.pool);
    const int j_lo = max(max(0, p - window + 1), a.chunk > 0 ? p / a.chunk * a.chunk : 0);
    const int n_keys = n_pool + (p - j_lo + 1);
    const int per = ((n_keys + n_split - 1) / n_split + kCgKeys - 1) / kCgKeys * kCgKeys, lo = split * per, hi = min(n_keys, lo + per);
    unsigned char* s_k = smem + w * z.warp_bytes;
    unsigned char* s_v = s_k + kCgKeys * z.ks16 * 16;
    const unsigned kaddr = (unsigned)__cvta_generic_to_shared(s_k), vaddr = (unsigned)__cvta_generic_to_shared(s_v);
    const __nv_bfloat16* own = (const __nv_bfloat16*)a.kv + (int64_t)t * v0.row_kv;

    // this lane's key of the tile at k0 (behind the run: the row itself, whose weight is then 0)
    auto row_of = [&](int k0) -> const __nv_bfloat16* {
        const int k = k0 + lane;
        if (k >= hi) return own;
        if (k < n_pool) return (const __nv_bfloat16*)a.pool_cache + ((int64_t)slot * a.pool_len + k) * v0.row_kv;
        const int j = j_lo + (k - n_pool);
        return j >= p ? own : (const __nv_bfloat16*)a.kv_cache + ((int64_t)slot * a.kv_len + j % a.kv_len) * v0.row_kv;
    };
    // the tile's keys or values: a row's 16-byte pieces side by side over the lanes, as many rows at a time as fit.  `even`: the
    // 32 rows lie one after the other behind the first (a tile of the ring without its end), so no lane has to be asked.
    auto fetch = [&](const __nv_bfloat16* row, bool even, int off, int n8, unsigned dst, int stride) {
        const int rpi = 32 / n8, r = lane / n8, c = lane - r * n8;          // (n8 <= 16)
        const unsigned out = dst + c * 16;
        if (even) {
            const __nv_bfloat16* src = (const __nv_bfloat16*)__shfl_sync(0xffffffffu, (unsigned long long)row, 0) + off + c * 8;
            if (r < rpi)
#pragma unroll 4
                for (int k = r; k < kCgKeys; k += rpi)
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(out + k * stride), "l"(src + (int64_t)k * v0.row_kv) : "memory");
        } else {
            for (int k = 0; k < kCgKeys; k += rpi) {
                const int kk = min(k + r, kCgKeys - 1);
                const __nv_bfloat16* src = (const __nv_bfloat16*)__shfl_sync(0xffffffffu, (unsigned long long)row, kk);
                if (r < rpi && k + r < kCgKeys)
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(out + kk * stride), "l"(src + off + c * 8) : "memory");
            }
        }
        __syncwarp();
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    auto is_even = [&](int k0) {
        const int j = j_lo + (k0 - n_pool);                                 // the first key's position
        return k0 >= n_pool && k0 + kCgKeys <= hi && j + kCgKeys <= p && j % a.kv_len + kCgKeys <= a.kv_len;
    };
    const int step = NW * kCgKeys;
    int k0 = lo + w * kCgKeys;
    if (k0 < hi) {
        const __nv_bfloat16* row = row_of(k0);
        const bool even = is_even(k0);
        fetch(row, even, v0.koff, dim / 8, kaddr, z.ks16 * 16);
        fetch(row, even, v0.voff, vdim / 8, vaddr, z.vs16 * 16);
    }
    if (dim % 16) *reinterpret_cast<uint4*>(s_k + lane * z.ks16 * 16 + dim * 2) = make_uint4(0, 0, 0, 0);      // the last k step's second half
    // rows of the products: head hr; a lane's places in a row's pairs of numbers: 2 qd, 2 qd + 1
    const int hr = lane >> 2, qd = lane & 3, h = h0 + min(hr, nh - 1), ksteps = (dim + 15) / 16, nvt = vdim / 8;
    uint32_t qa[8][2];
    const __nv_bfloat16* qrow = (const __nv_bfloat16*)a.q + (int64_t)t * v0.qstride + h * dim;
#pragma unroll
    for (int ks = 0; ks < 8; ++ks)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int d = ks * 16 + e * 8 + qd * 2;
            qa[ks][e] = hr < nh && d < dim ? *reinterpret_cast<const uint32_t*>(qrow + d) : 0u;
        }
    const float hb = MODE == UMBS_ATTN_SIGMOID && a.head_bias ? a.head_bias[h] : 0.f;
    const float r1h = a.r1 ? a.r1[h] : 0.f, r2h = a.r1 ? a.r2[h] : 0.f;
    float m = -INFINITY, l = 0.f, o[16][2];
#pragma unroll
    for (int j = 0; j < 16; ++j) o[j][0] = o[j][1] = 0.f;
    for (; k0 < hi; k0 += step) {
        const bool more = k0 + step < hi, even = more && is_even(k0 + step);
        const __nv_bfloat16* next = more ? row_of(k0 + step) : own;
        asm volatile("cp.async.wait_group 1;" ::: "memory");                // the keys are here (the values may not be)
        __syncwarp();
        float sc[4][2] = {};
#pragma unroll
        for (int kp = 0; kp < 4; ++kp) {
            if (kp * 2 >= ksteps) break;
#pragma unroll
            for (int nt = 0; nt < 4; ++nt) {
                uint32_t r[4];
                ldsm4(r, kaddr + (nt * 8 + (lane & 7)) * z.ks16 * 16 + kp * 64 + (lane >> 3) * 16);
                float d[2][4] = {};
                mma_top(d[0], qa[2 * kp][0], qa[2 * kp][1], r[0], r[1]);
                if (2 * kp + 1 < ksteps) mma_top(d[1], qa[2 * kp + 1][0], qa[2 * kp + 1][1], r[2], r[3]);
                sc[nt][0] += d[0][0] + d[1][0];
                sc[nt][1] += d[0][1] + d[1][1];
            }
        }
        __syncwarp();
        if (more) fetch(next, even, v0.koff, dim / 8, kaddr, z.ks16 * 16);  // (the key tile has been read)
        else asm volatile("cp.async.commit_group;" ::: "memory");
        float pw[4][2];
        float mx = -INFINITY;
#pragma unroll
        for (int nt = 0; nt < 4; ++nt)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int k = k0 + nt * 8 + qd * 2 + e;
                if (MODE == UMBS_ATTN_SIGMOID) {
                    pw[nt][e] = k < hi ? sigmoidf_(sc[nt][e] * a.scale + hb) : 0.f;
                } else {
                    pw[nt][e] = k < hi ? shaped_score(a, sc[nt][e], r1h, r2h, k < n_pool ? 0 : p - (j_lo + k - n_pool)) : -INFINITY;
                    mx = fmaxf(mx, pw[nt][e]);
                }
            }
        if (MODE != UMBS_ATTN_SIGMOID) {
            mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
            mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
            const float mn = fmaxf(m, mx), ref = mn > -INFINITY ? mn : 0.f, corr = expf(m - ref);      // (m = -inf the first time: corr = 0)
            float ls = 0.f;
#pragma unroll
            for (int nt = 0; nt < 4; ++nt)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    pw[nt][e] = expf(pw[nt][e] - ref);
                    ls += pw[nt][e];
                }
            l = l * corr + ls;                                              // (a lane's own keys; added up at the end)
            m = mn;
            if (__any_sync(0xffffffffu, corr != 1.f)) {
#pragma unroll
                for (int j = 0; j < 16; ++j) {
                    o[j][0] *= corr;
                    o[j][1] *= corr;
                }
            }
        }
        // the weights' three parts as row fragments of the second product, for keys 0-15 and 16-31
        uint32_t pa[3][2][2];
#pragma unroll
        for (int nt = 0; nt < 4; ++nt) {
            float x = pw[nt][0], y = pw[nt][1];
#pragma unroll
            for (int e = 0; e < 3; ++e) {
                pa[e][nt >> 1][nt & 1] = __byte_perm(__float_as_uint(x), __float_as_uint(y), 0x7632);
                x -= __uint_as_float(__float_as_uint(x) & 0xffff0000u);
                y -= __uint_as_float(__float_as_uint(y) & 0xffff0000u);
            }
        }
        asm volatile("cp.async.wait_group 1;" ::: "memory");                // the values
        __syncwarp();
#pragma unroll
        for (int j = 0; j < 16; ++j) {
            if (j >= nvt) break;
            uint32_t r[4];
            ldsm4t(r, vaddr + lane * z.vs16 * 16 + j * 16);
            float d[4] = {};
#pragma unroll
            for (int e = 2; e >= 0; --e) {
                mma_top(d, pa[e][0][0], pa[e][0][1], r[0], r[1]);
                mma_top(d, pa[e][1][0], pa[e][1][1], r[2], r[3]);
            }
            o[j][0] += d[0];
            o[j][1] += d[1];
        }
        __syncwarp();
        if (more) fetch(next, even, v0.voff, vdim / 8, vaddr, z.vs16 * 16);
        else asm volatile("cp.async.commit_group;" ::: "memory");
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    // merge: the warps' triples over the tiles' memory
    float* s_o = reinterpret_cast<float*>(smem);                            // [warps][heads][vdim]
    float* s_ml = s_o + NW * kCgHeads * vdim;                         // [warps][heads][2]
    l += __shfl_xor_sync(0xffffffffu, l, 1);
    l += __shfl_xor_sync(0xffffffffu, l, 2);
#pragma unroll
    for (int j = 0; j < 16; ++j)
        if (j < nvt) *reinterpret_cast<float2*>(s_o + (w * kCgHeads + hr) * vdim + j * 8 + qd * 2) = make_float2(o[j][0], o[j][1]);
    if (qd == 0) { s_ml[(w * kCgHeads + hr) * 2] = m; s_ml[(w * kCgHeads + hr) * 2 + 1] = l; }
    float odd = 0.f;                                                        // stays 0 while the sums are finite
#pragma unroll
    for (int j = 0; j < 16; ++j) odd = fmaf(o[j][0], 0.f, fmaf(o[j][1], 0.f, odd));
    if (__any_sync(0xffffffffu, hr < nh && odd != 0.f)) {
        __syncwarp();
        for (int g = 0; g < nh; ++g)
            plain_part<MODE, NW>(a, v0, (const __nv_bfloat16*)a.q + (int64_t)t * v0.qstride + (h0 + g) * dim, h0 + g, own, slot, p, n_pool, j_lo,
                             lo + w * kCgKeys, hi, s_o + (w * kCgHeads + g) * vdim, s_ml + (w * kCgHeads + g) * 2);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < nh * vdim; i += 32 * NW) {
        const int g = i / vdim, c = i - g * vdim, hh = h0 + g;
        float Mx = -INFINITY, L = 0.f, O = 0.f;
        if (MODE == UMBS_ATTN_SIGMOID) {
            for (int ww = 0; ww < NW; ++ww) O += s_o[(ww * kCgHeads + g) * vdim + c];
        } else {
            const float sk = (n_split == 1 && MODE == UMBS_ATTN_SOFTMAX_SINK) ? sink_score(a, hh) : -INFINITY;
            for (int ww = 0; ww < NW; ++ww) Mx = fmaxf(Mx, s_ml[(ww * kCgHeads + g) * 2]);
            Mx = fmaxf(Mx, sk);
            for (int ww = 0; ww < NW; ++ww) {
                const float mw = s_ml[(ww * kCgHeads + g) * 2], f = mw > -INFINITY ? expf(mw - Mx) : 0.f;
                L = fmaf(s_ml[(ww * kCgHeads + g) * 2 + 1], f, L);
                O = fmaf(s_o[(ww * kCgHeads + g) * vdim + c], f, O);
            }
            if (n_split == 1 && MODE == UMBS_ATTN_SOFTMAX_SINK) L += expf(sk - Mx);
        }
        if (n_split > 1) {
            float* pr = part + (((int64_t)t * a.heads + hh) * n_split + split) * (vdim + 2);
            pr[c] = O;
            if (c == 0) { pr[vdim] = Mx; pr[vdim + 1] = L; }
            continue;
        }
        const float inv = MODE == UMBS_ATTN_SIGMOID ? 1.f : 1.f / L;
        float gt = 1.f;
        if (a.gate) gt = sigmoidf_(a.gate[(int64_t)t * a.ldg + (a.gate_per_head ? hh : hh * vdim + c)]);
        ((__nv_bfloat16*)a.out)[(int64_t)t * a.heads * vdim + (int64_t)hh * vdim + c] = __float2bfloat16_rn(O * inv * gt);
    }
}

// One block per (token, head): the splits' triples, in split order, then the sink, the division and the output gate.
template <typename T, int MODE>
__global__ void cached_attention_merge_kernel(CachedAttnArgs a, int n_split, const float* __restrict__ part) {
    chain_wait();
    const int nv = a.heads * a.maps * a.vheads;
    const int th = blockIdx.x, t = th / nv, h = th - t * nv, vdim = a.vdim, c = threadIdx.x;      // (without options h is the head)
    const float* pr = part + (int64_t)th * n_split * (vdim + 2);
    const float sk = MODE == UMBS_ATTN_SOFTMAX_SINK ? sink_score(a, h / (a.maps * a.vheads)) : -INFINITY;
    float M = sk, L = 0.f, O = 0.f;
    if (MODE == UMBS_ATTN_SIGMOID) {
        if (c < vdim)
            for (int i = 0; i < n_split; ++i) O += pr[i * (vdim + 2) + c];
    } else {
        for (int i = 0; i < n_split; ++i) M = fmaxf(M, pr[i * (vdim + 2) + vdim]);
        for (int i = 0; i < n_split; ++i) {
            const float mi = pr[i * (vdim + 2) + vdim], f = mi > -INFINITY ? expf(mi - M) : 0.f;
            L = fmaf(pr[i * (vdim + 2) + vdim + 1], f, L);
            if (c < vdim) O = fmaf(pr[i * (vdim + 2) + c], f, O);
        }
        if (MODE == UMBS_ATTN_SOFTMAX_SINK) L += expf(sk - M);
    }
    if (c < vdim) {
        const float inv = MODE == UMBS_ATTN_SIGMOID ? 1.f : 1.f / L;
        if (a.raw != nullptr) { a.raw[(int64_t)th * vdim + c] = O * inv; return; }
        float gt = 1.f;
        if (a.gate) gt = sigmoidf_(a.gate[(int64_t)t * a.ldg + (a.gate_per_head ? h : h * vdim + c)]);
        ((T*)a.out)[(int64_t)t * a.heads * vdim + (int64_t)h * vdim + c] = from_f32<T>(O * inv * gt);
    }
}

template <typename T, int MODE>
static int launch_decode(const CachedAttnArgs& a, const Batch& b, int n_split, float* part, cudaStream_t st) {
    const int nv = a.heads * a.maps * a.vheads;
    chain_launch(cached_attention_decode_kernel<T, MODE>, dim3(n_split, nv, b.n_seqs), 32 * kCdWarps, 0, st, a, b, n_split, part);
    if (n_split > 1) chain_launch(cached_attention_merge_kernel<T, MODE>, b.n_tokens * nv, a.vdim <= 128 ? 128 : 256, 0, st, a, n_split, part);
    return 0;
}

// Sizes the grouped kernel takes: rows in 16-byte pieces, at most 128 numbers (eight k steps, sixteen value tiles in registers).
// fp32 results stay with the fp32 kernel: at 64 dimensions its error to float64 is 2.2e-7, the tensor path's 2.9e-7.
static bool group_fits(const CachedAttnArgs& a) {
    auto al = [](const void* q) { return ((uintptr_t)q & 15) == 0; };
    return a.raw == nullptr && a.dim % 8 == 0 && a.vdim % 8 == 0 && a.dim <= 128 && a.vdim <= 128 && al(a.q) && al(a.kv) && al(a.kv_cache) &&
           (a.pool <= 0 || al(a.pool_cache));
}
// Few keys: a block of the grouped kernel is a chain of copies and products as long for one key as for 128, 6 us at 64 dimensions and
// 8 at 128; a block per head takes 4 us for up to 32 keys and 2 for every 32 more, while its blocks are few (16 heads over 4 of
// 128, us per head / grouped: 8 sequences of 11 keys 4.3 / 8.4, of 64 6.9 / 8.2, of 81 8.4 / 8.2; 32 of 11 8.0 / 8.4; 64 of 11 13.7 / 9.0; heads on their
// own, 64 sequences of 21 keys: 8.6 / 14.5).  A captured step keeps the grouped kernel: its graph is replayed for longer contexts.
static bool few_keys(const CachedAttnArgs& a, int keys, int rows) {
    if (a.heads == a.kv_heads && keys <= 32) return true;
    if (a.dim > 64 && rows <= 512 && keys <= 16) return true;
    return rows <= 256 && keys <= (a.dim > 64 ? 64 : 32);
}
static bool capturing(cudaStream_t st) {
    cudaStreamCaptureStatus s = cudaStreamCaptureStatusNone;
    return cudaStreamIsCapturing(st, &s) != cudaSuccess || s != cudaStreamCaptureStatusNone;
}
// Unsplit steps of a block per SM and more may take blocks of six warps (six_warps_pay: waves against rounds): what bounds a block is the chain of a warp's rounds (issue
// slots 33 %, with six warps 40 %), and with two blocks of four warps on an SM 1040 keys are nine of them, with six warps six.  us, four warps / six, fewer blocks, 16
// heads over 4 of 128: 32 x 256 10.6 and a merge / 13.5, 8 x 1024 10.5 / 11.4, 1 x 4096 10.0 / 11.2.
constexpr int kCgSms = 148;
static int group_blocks(const CachedAttnArgs& a) {
    return a.kv_heads * ((a.heads / a.kv_heads + kCgHeads - 1) / kCgHeads);
}

template <int MODE, int NW>
static int launch_group(const CachedAttnArgs& a, const Batch& b, int n_split, float* part, cudaStream_t st) {
    const int tiles = NW * group_sizes(a.dim, a.vdim).warp_bytes, merge = NW * kCgHeads * (a.vdim + 2) * 4, smem = tiles > merge ? tiles : merge;
    auto kernel = cached_attention_decode_group_kernel<MODE, NW>;
    if (smem > 48 * 1024) {                                 // (always the same limit: another thread may be between setting it and its launch)
        const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, NW * group_sizes(128, 128).warp_bytes);
        if (e != cudaSuccess) return (int)e;
    }
    // (one or two blocks to an SM: brought in while the means in front of them end, they fall on the SMs unevenly, 60 -> 62 us of 64
    // sequences; in a model's step the kernel in front is over sooner)
    chain_launch_if(in_chain(), kernel, dim3(n_split, group_blocks(a), b.n_seqs), 32 * NW, smem, st, a, b, n_split, part);
    if (n_split > 1) chain_launch(cached_attention_merge_kernel<__nv_bfloat16, MODE>, b.n_tokens * a.heads, a.vdim <= 128 ? 128 : 256, 0, st, a, n_split, part);
    return 0;
}
template <int NW>
static int launch_group_any(int mode, const CachedAttnArgs& a, const Batch& b, int n_split, float* part, cudaStream_t st) {
    switch (mode) {
        case UMBS_ATTN_SOFTMAX: return launch_group<UMBS_ATTN_SOFTMAX, NW>(a, b, n_split, part, st);
        case UMBS_ATTN_SOFTMAX_SINK: return launch_group<UMBS_ATTN_SOFTMAX_SINK, NW>(a, b, n_split, part, st);
        case UMBS_ATTN_SIGMOID: return launch_group<UMBS_ATTN_SIGMOID, NW>(a, b, n_split, part, st);
    }
    return UMB_ERR_ARG;
}

template <typename T>
static int launch_decode_any(int mode, const CachedAttnArgs& a, const Batch& b, int n_split, float* part, cudaStream_t st) {
    switch (mode) {
        case UMBS_ATTN_SOFTMAX: return launch_decode<T, UMBS_ATTN_SOFTMAX>(a, b, n_split, part, st);
        case UMBS_ATTN_SOFTMAX_SINK: return launch_decode<T, UMBS_ATTN_SOFTMAX_SINK>(a, b, n_split, part, st);
        case UMBS_ATTN_SIGMOID: return launch_decode<T, UMBS_ATTN_SIGMOID>(a, b, n_split, part, st);
    }
    return UMB_ERR_ARG;
}

}  // namespace umbs

using namespace umbs;

namespace umbs {
// One warp per (token, head): from the virtual heads' raw outputs to the head's output.
template <typename T>
__global__ void attention_finish_kernel(const float* __restrict__ raw, int n_pairs, int heads, int kv_heads, int vdim, int maps,
                                        int vheads, const float* __restrict__ talk, float lambda, int unit_norm, float eps,
                                        float out_mult, const float* __restrict__ gate, int64_t ldg, T* __restrict__ out) {
    const int pair = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (pair >= n_pairs) return;
    const int t = pair / heads, h = pair - t * heads, nv = heads * maps * vheads;
    const float* rt = raw + (int64_t)t * nv * vdim;
    float v[8], ss = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int c = lane + 32 * i;
        v[i] = 0.f;
        if (c >= vdim) continue;
        if (talk != nullptr) {
            const int own = h / (heads / kv_heads);                       // the value head of query head h
            float acc = 0.f;
            for (int g = 0; g < heads; ++g) acc = fmaf(talk[h * heads + g], rt[(int64_t)(g * vheads + own) * vdim + c], acc);
            v[i] = acc;
        } else if (maps == 2) {
            v[i] = rt[(int64_t)(h * 2) * vdim + c] - lambda * rt[(int64_t)(h * 2 + 1) * vdim + c];
        } else {
            v[i] = rt[(int64_t)h * vdim + c];
        }
        ss = fmaf(v[i], v[i], ss);
    }
#pragma unroll
    for (int x = 16; x > 0; x >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, x);
    const float f = (unit_norm ? 1.f / sqrtf(ss / (float)vdim + eps) : 1.f) * out_mult;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int c = lane + 32 * i;
        if (c >= vdim) continue;
        float o = v[i] * f;
        if (gate != nullptr) o *= sigmoidf_(gate[(int64_t)t * ldg + h * vdim + c]);
        out[(int64_t)t * heads * vdim + h * vdim + c] = from_f32<T>(o);
    }
}

}  // namespace umbs

extern "C" int umbs_attention_finish(int dtype, const float* raw, int n_tokens, int heads, int kv_heads, int vdim, int maps,
                                     int value_heads, const float* talk, float diff_lambda, int unit_norm, float eps,
                                     float out_mult, const float* gate, int64_t ldg, void* out, umbs_stream_t stream) {
    if (n_tokens <= 0) return 0;
    maps = maps < 1 ? 1 : maps;
    value_heads = value_heads < 1 ? 1 : value_heads;
    if (raw == nullptr || out == nullptr || heads < 1 || kv_heads < 1 || heads % kv_heads != 0) return UMB_ERR_ARG;
    if (vdim < 1 || vdim > 256 || maps > 2) return UMB_ERR_UNSUPPORTED;
    if (talk != nullptr ? (maps != 1 || value_heads != kv_heads) : value_heads != 1) return UMB_ERR_UNSUPPORTED;
    cudaStream_t st = (cudaStream_t)stream;
    const int pairs = n_tokens * heads;
    if (dtype == UMBS_BF16)
        attention_finish_kernel<__nv_bfloat16><<<(pairs + 3) / 4, 128, 0, st>>>(raw, pairs, heads, kv_heads, vdim, maps, value_heads, talk,
                                                                               diff_lambda, unit_norm, eps, out_mult != 0.f ? out_mult : 1.f,
                                                                               gate, ldg, (__nv_bfloat16*)out);
    else if (dtype == UMBS_F32)
        attention_finish_kernel<float><<<(pairs + 3) / 4, 128, 0, st>>>(raw, pairs, heads, kv_heads, vdim, maps, value_heads, talk, diff_lambda,
                                                                       unit_norm, eps, out_mult != 0.f ? out_mult : 1.f, gate, ldg, (float*)out);
    else return UMB_ERR_ARG;
    count_launches(1);
    return (int)cudaGetLastError();
}

extern "C" int umbs_cached_attention(int dtype, int mode, const void* q, const void* kv, const void* kv_cache, int kv_len,
                                     const void* pool_cache, int pool_len, const umbs_batch_t* batch, int heads,
                                     int kv_heads, int dim, int vdim, int window, int pool, float scale,
                                     const float* head_bias, const float* gate, int64_t ldg, int gate_per_head,
                                     float* split_scratch, size_t split_bytes, void* out, umbs_stream_t stream) {
    return umbs_cached_attention_ex(dtype, mode, q, kv, kv_cache, kv_len, pool_cache, pool_len, batch, heads, kv_heads, dim, vdim,
                                    window, pool, scale, head_bias, gate, ldg, gate_per_head, nullptr, split_scratch, split_bytes,
                                    out, stream);
}

extern "C" int umbs_cached_attention_ex(int dtype, int mode, const void* q, const void* kv, const void* kv_cache, int kv_len,
                                        const void* pool_cache, int pool_len, const umbs_batch_t* batch, int heads,
                                        int kv_heads, int dim, int vdim, int window, int pool, float scale,
                                        const float* head_bias, const float* gate, int64_t ldg, int gate_per_head,
                                        const umbs_attn_opts_t* opts, float* split_scratch, size_t split_bytes, void* out,
                                        umbs_stream_t stream) {
    if (batch->n_tokens <= 0) return 0;
    if (heads < 1 || kv_heads < 1 || heads % kv_heads != 0 || kv_len < 1) return UMB_ERR_ARG;
    if (pool > 0 && (window <= 0 || pool_cache == nullptr || pool_len < 1)) return UMB_ERR_ARG;
    if (dim < 1 || vdim < 1 || dim > 256 || vdim > 256) return UMB_ERR_UNSUPPORTED;      // tiles and lanes are sized for heads up to 256
    cudaStream_t st = (cudaStream_t)stream;
    CachedAttnArgs a{q, kv, kv_cache, pool_cache, kv_len, pool_len, heads, kv_heads, dim, vdim, window, pool, scale,
                     head_bias, gate, ldg, gate_per_head, out, 0.f, nullptr, nullptr, 0, 1, 1, nullptr, nullptr};
    if (opts != nullptr) {
        a.softcap = opts->softcap; a.r1 = opts->dist_r1; a.r2 = opts->dist_r2; a.chunk = opts->chunk;
        a.maps = opts->maps > 0 ? opts->maps : 1; a.vheads = opts->value_heads > 0 ? opts->value_heads : 1; a.raw = opts->raw_out;
        a.sink = opts->sink;
        const bool any = a.softcap > 0.f || a.r1 != nullptr || a.chunk > 0 || a.maps > 1 || a.vheads > 1;
        if ((a.r1 != nullptr) != (a.r2 != nullptr) || a.chunk < 0) return UMB_ERR_ARG;
        if (any && (pool > 0 || mode == UMBS_ATTN_SIGMOID)) return UMB_ERR_UNSUPPORTED;
        if ((a.maps > 1 || a.vheads > 1) && a.raw == nullptr) return UMB_ERR_ARG;      // several rows per head need the finishing pass
        if (a.vheads != 1 && a.vheads != kv_heads) return UMB_ERR_ARG;
    }
    if (a.raw == nullptr && out == nullptr) return UMB_ERR_ARG;
    heads = a.heads * a.maps * a.vheads;                   // rows per token from here on (splits, scratch)
    int rc;
    if (batch->max_seq_len == 1) {
        // a decode step: about 256 keys per block, as many splits as the longest context of the step asks for, the GPU
        // has room for (two blocks per SM) and the scratch buffer holds
        int keys = window > 0 ? (batch->max_pos0 < window ? batch->max_pos0 + 1 : window + (pool > 0 ? batch->max_pos0 / pool : 0))
                              : batch->max_pos0 + 1;
        if (a.chunk > 0 && keys > a.chunk) keys = a.chunk;
        const int rows = batch->n_seqs * heads;
        const bool group = dtype == UMBS_BF16 && group_fits(a) && !(few_keys(a, keys, rows) && !capturing(st));
        const size_t per_split = (size_t)rows * (vdim + 2) * sizeof(float);
        const int room = split_scratch == nullptr || per_split == 0 ? 1 : (int)std::clamp<size_t>(split_bytes / per_split, 1, 32);
        int n_split = 1;
        bool group_many = false;
        if (group) {
            // heads that share a key/value head in one block, three blocks on an SM, 128 keys a round of its warps: the split with
            // the fewest rounds from first to last block, one more per block for its start and end
            const int64_t blocks = (int64_t)batch->n_seqs * group_blocks(a);
            int64_t best = INT64_MAX;
            for (int n = 1; n <= room && (n == 1 || (n - 1) * 128 < keys); ++n) {
                const int64_t cost = (blocks * n + 3 * kCgSms - 1) / (3 * kCgSms) * ((keys + n * 128 - 1) / (n * 128) + 1) + (n > 1);
                if (cost < best) { best = cost; n_split = n; }
            }
            // (a captured step is replayed for longer contexts: by the most that its ring and its window hold)
            const int most = std::max(keys, std::min(kv_len, window > 0 ? window : kv_len));
            group_many = n_split == 1 && umb::six_warps_pay(blocks, keys, kCgSms);
            if (n_split == 1 && group_many != umb::six_warps_pay(blocks, most, kCgSms) && capturing(st)) group_many = !group_many;
        } else {
            n_split = (keys + 255) / 256;
            n_split = n_split < 1 ? 1 : (n_split > 32 ? 32 : n_split);
            n_split = std::min(n_split, std::min((296 + rows - 1) / rows, room));
        }
        if (group) rc = (group_many ? launch_group_any<6> : launch_group_any<4>)(mode, a, *batch, n_split, split_scratch, st);
        else if (dtype == UMBS_BF16) rc = launch_decode_any<__nv_bfloat16>(mode, a, *batch, n_split, split_scratch, st);
        else if (dtype == UMBS_F32) rc = launch_decode_any<float>(mode, a, *batch, n_split, split_scratch, st);
        else return UMB_ERR_ARG;
        if (rc) return rc;
        count_launches(n_split > 1 ? 2 : 1);
        return (int)cudaGetLastError();
    }
    if (dtype == UMBS_BF16 && attention_tc_fits(a, nullptr)) rc = launch_attention_tc(mode, a, nullptr, *batch, st);
    else if (dtype == UMBS_BF16) rc = launch_any<__nv_bfloat16>(mode, a, *batch, st);
    else if (dtype == UMBS_F32) rc = launch_any<float>(mode, a, *batch, st);
    else return UMB_ERR_ARG;
    if (rc) return rc;
    count_launches(1);
    return (int)cudaGetLastError();
}
