// Matrix products of the sequence-state decoders: C = A W^T with W stored [out, in], batched over groups (heads or
// experts), optionally over expert-sorted gathered rows, optionally with the gated feed-forward activation fused
// into the epilogue of a gate|up pair of products.
//
// Five kernels share one argument block:
//   * gemm_simt_kernel  -- fp32 FMA chains over shared-memory tiles: every shape that the others do not take (unaligned rows; bf16
//                          with K not a multiple of 32);
//   * gemm_split_kernel -- fp32 operands (true 32-bit) as sums of bf16 numbers through tcgen05 (seq_gemm_split.cu);
//   * gemm_tc_kernel    -- bf16 operands through tcgen05 with fp32 accumulators (seq_gemm_tc.cu);
//   * gemm_skinny_kernel, gemm_rows_kernel -- few rows (decoding), bf16 and fp32: a weight stream with the rows' partial sums in
//                          registers.
// In each of them the order in which an output element's products are added up (one chain, or shares of k by themselves first) does not
// depend on the other rows, so a row's result is the same whatever else is in the batch; which kernel runs depends on the row count and
// the alignment, and they differ from each other by rounding only.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <algorithm>

#include "seq_gemm.h"

namespace umbs {

// ------------------------------------------------------------------------------------------------ SIMT
// 64 x 64 outputs per block of 64 threads, 8 x 8 a thread (or, for small products, 16 x 64 and 2 x 8; with DUAL: 8 rows x 4 gate and the same 4 up columns), k in steps of
// 16 through two shared-memory stages, the next step's numbers on their way in registers.  Per k a thread reads four 16-byte
// pieces for 64 multiply-adds, two of them an instruction; an output is one chain of additions over k, so it has the same bits
// in every tiling.  Bound: two warps a scheduler (162 registers) that wait on their own
// chains: issue slots 39 % taken, shared memory 52 %, 2.7 times the time of the multiply-adds alone.  Blocks are small so that a step of some hundred rows spreads evenly: 777 x 1024
// -> 3088 are 637 of them: 178 us (27.6 TFLOP/s) as fp32 with rows that the tensor-core form does not take.
constexpr int BN = 64, BK = 16;

template <typename T> __device__ __forceinline__ void load_k4(const T* p, int left, bool vec, float (&f)[4]) {
#pragma unroll
    for (int i = 0; i < 4; ++i) f[i] = i < left ? to_f32(p[i]) : 0.f;
}
template <> __device__ __forceinline__ void load_k4<float>(const float* p, int left, bool vec, float (&f)[4]) {
    if (vec && left >= 4) {
        const float4 v = *reinterpret_cast<const float4*>(p);
        f[0] = v.x; f[1] = v.y; f[2] = v.z; f[3] = v.w;
    } else {
#pragma unroll
        for (int i = 0; i < 4; ++i) f[i] = i < left ? p[i] : 0.f;
    }
}

template <typename TA, typename TC, bool DUAL, int RT>
__global__ void __launch_bounds__(64) gemm_simt_kernel(GemmArgs a, int vec, int vec_c) {
    constexpr int BM = 8 * RT, LA = BM / 16;                // RT rows a thread; LA: rows of A a thread loads
    __shared__ __align__(16) float As[2][BK][BM + 4], Ws[2][BK][BN + 4];
    const int g = blockIdx.z;
    int row_lo = 0, rows = a.M;
    if (a.grp_off != nullptr) { row_lo = a.grp_off[g]; rows = a.grp_off[g + 1] - row_lo; }
    constexpr int OUT = DUAL ? BN / 2 : BN;                 // output columns of a block
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * OUT;
    if (m0 >= rows) return;
    const TA* A = (const TA*)a.A + (int64_t)g * a.a_goff;
    const TA* W = (const TA*)a.W + (int64_t)g * a.w_gstride;
    const int tid = threadIdx.x, tx = tid & 7, ty = tid >> 3;
    // loader: a thread takes four k of rows lr, lr + 16, lr + 32, lr + 48 of both tiles
    const int lr = tid >> 2, lk = (tid & 3) * 4;
    const TA *ap[LA], *wp[4];
#pragma unroll
    for (int i = 0; i < LA; ++i) {
        const int r = lr + 16 * i, p = row_lo + m0 + r;
        ap[i] = m0 + r < rows ? A + (int64_t)(a.row_src ? a.row_src[p] : p) * a.lda + lk : nullptr;
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int r = lr + 16 * i;
        wp[i] = nullptr;
        const int n = n0 + (DUAL ? r % OUT : r);            // (DUAL: 32 gate rows, then the 32 up rows)
        if (n < a.N) wp[i] = W + (int64_t)(DUAL && r >= OUT ? a.N + n : n) * a.ldw + lk;
    }
    float ra[LA][4], rw[4][4];
    auto fetch = [&](int k0) {
        const int left = a.K - k0 - lk;
#pragma unroll
        for (int i = 0; i < LA; ++i) load_k4<TA>(ap[i] + k0, ap[i] != nullptr ? left : 0, vec, ra[i]);
#pragma unroll
        for (int i = 0; i < 4; ++i) load_k4<TA>(wp[i] + k0, wp[i] != nullptr ? left : 0, vec, rw[i]);
    };
    auto stash = [&](int st) {
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                if (i < LA) As[st][lk + e][lr + 16 * i] = ra[i < LA ? i : 0][e];
                Ws[st][lk + e][lr + 16 * i] = rw[i][e];
            }
    };
    f32x2 acc[RT][4] = {};                                  // rows ty 4 .. + 3 and 32 + ty 4 .. (RT = 2: 2 ty, + 1); columns tx 4 .. + 3 and 32 + tx 4 .., in pairs
    fetch(0);
    stash(0);
    __syncthreads();
    int st = 0;
    for (int k0 = 0; k0 < a.K; k0 += BK, st ^= 1) {
        const bool more = k0 + BK < a.K;
        if (more) fetch(k0 + BK);
#pragma unroll
        for (int k = 0; k < BK; ++k) {
            float av[RT];
            if constexpr (RT == 8) {
                *reinterpret_cast<float4*>(av) = *reinterpret_cast<const float4*>(&As[st][k][ty * 4]);
                *reinterpret_cast<float4*>(av + 4) = *reinterpret_cast<const float4*>(&As[st][k][32 + ty * 4]);
            } else {
                *reinterpret_cast<float2*>(av) = *reinterpret_cast<const float2*>(&As[st][k][ty * 2]);
            }
            const ulonglong2 w0 = *reinterpret_cast<const ulonglong2*>(&Ws[st][k][tx * 4]), w1 = *reinterpret_cast<const ulonglong2*>(&Ws[st][k][32 + tx * 4]);
#pragma unroll
            for (int i = 0; i < RT; ++i) {
                const f32x2 aa = pack2(av[i], av[i]);
                acc[i][0] = fma2(aa, w0.x, acc[i][0]);
                acc[i][1] = fma2(aa, w0.y, acc[i][1]);
                acc[i][2] = fma2(aa, w1.x, acc[i][2]);
                acc[i][3] = fma2(aa, w1.y, acc[i][3]);
            }
        }
        if (more) {
            stash(st ^ 1);                                  // the other stage was last read in front of the barrier before
            __syncthreads();
        }
    }
    TC* C = (TC*)a.C + (int64_t)g * a.c_goff;
#pragma unroll
    for (int i = 0; i < RT; ++i) {
        const int m = m0 + (RT == 8 ? (i >> 2) * 32 + ty * 4 + (i & 3) : ty * 2 + i);
        if (m >= rows) continue;
#pragma unroll
        for (int half = 0; half < (DUAL ? 1 : 2); ++half) {
            const int n = n0 + half * 32 + tx * 4;
            if (n >= a.N) continue;
            const float2 u0 = unpack2(acc[i][half * 2]), u1 = unpack2(acc[i][half * 2 + 1]), p0 = unpack2(acc[i][2]), p1 = unpack2(acc[i][3]);
            const float s1[4] = {u0.x, u0.y, u1.x, u1.y}, s2[4] = {p0.x, p0.y, p1.x, p1.y};
            float v[4];
#pragma unroll
            for (int e = 0; e < 4; ++e)
                if (n + e < a.N) v[e] = finish<DUAL>(a, s1[e], DUAL ? s2[e] : 0.f, g, row_lo + m, n + e);
            TC* out = C + (int64_t)(row_lo + m) * a.ldc + n;
            if (sizeof(TC) == 4 && vec_c && n + 4 <= a.N) {
                *reinterpret_cast<float4*>(out) = make_float4(v[0], v[1], v[2], v[3]);
            } else {
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    if (n + e < a.N) out[e] = from_f32<TC>(v[e]);
            }
        }
    }
}

// ------------------------------------------------------------------------------------------------ few rows (decode)
// Up to 16 bf16 activation rows per group: the product is a stream over the weights.  A warp owns R weight rows (with DUAL: R / 2 gate
// rows and their up rows) and a share of k.  mma.m16n8k16 takes the weights as its 16-row operand and the activations as its 8-column
// one, or (R = 8) the other way round.  Which k sits where in a product does not matter as long as both operands agree, so a lane
// fetches 8 V neighbouring k of its weight rows and of its activation rows, straight into the registers that the products read, and U
// such steps are in flight before the first is used.  KW warps of a block share a tile's k.
// Sums: every product starts from zero, a step's products are added in fp32 pair by pair, the steps in order, the warps in fp64: no chain
// runs through the tensor core, which cuts its sums off (5 to 7e-8 from float64 for K = 384 to 4096, 6 to 8e-8 as chains of
// multiply-adds).  The order depends on the weight's sizes and on whether rows start on 32 bytes or 16 (launch_skinny): a row's result does not
// depend on the other rows.  A group without rows returns before touching its weights, so a decode step reads only the experts that were chosen.
// Bound: a launch, a load's way from HBM and the reduction, one after the other: 8 rows of 2048 to 6144 columns 14.8 -> 6.7 us (3.8 TB/s;
// the multiply-adds that this replaced unpacked every weight for every row), of 1024 to 1024 3.9 -> 2.5, 16 rows 23.9 -> 9.3.
// V 16-byte pieces that follow one another: weights, which no other block reads, and activations
template <int V> __device__ __forceinline__ void load_weights(uint4 (&v)[V], const __nv_bfloat16* p) {
    if constexpr (V == 2)
        asm volatile("ld.global.nc.L1::no_allocate.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                     : "=r"(v[0].x), "=r"(v[0].y), "=r"(v[0].z), "=r"(v[0].w), "=r"(v[1].x), "=r"(v[1].y), "=r"(v[1].z), "=r"(v[1].w) : "l"(p));
    else
        asm volatile("ld.global.nc.L1::no_allocate.v4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(v[0].x), "=r"(v[0].y), "=r"(v[0].z), "=r"(v[0].w) : "l"(p));
}
template <int V> __device__ __forceinline__ void load_rows(uint4 (&v)[V], const __nv_bfloat16* p) {
    if constexpr (V == 2)
        asm volatile("ld.global.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                     : "=r"(v[0].x), "=r"(v[0].y), "=r"(v[0].z), "=r"(v[0].w), "=r"(v[1].x), "=r"(v[1].y), "=r"(v[1].z), "=r"(v[1].w) : "l"(p));
    else
        v[0] = *reinterpret_cast<const uint4*>(p);
}
__device__ __forceinline__ void mma_16816(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

template <typename TC, bool DUAL, int R, int NT, int KW, int U, int V>
__global__ void __launch_bounds__(32 * KW) gemm_skinny_kernel(const GemmArgs a) {
    constexpr int OUT = DUAL ? R / 2 : R, WR = R / 8;       // output columns of a block; weight rows of a lane
    __shared__ float part[KW][NT * 8][R + 1];
    const int g = blockIdx.y, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, q = lane >> 2, k8 = (lane & 3) * 8 * V, n0 = blockIdx.x * OUT;
    const __nv_bfloat16* A = (const __nv_bfloat16*)a.A + (int64_t)g * a.a_goff;
    const __nv_bfloat16* W = (const __nv_bfloat16*)a.W + (int64_t)g * a.w_gstride;
    const __nv_bfloat16 *w[WR], *x[NT];                     // rows q and q + 8 of the tile, of the activations
#pragma unroll
    for (int i = 0; i < WR; ++i) {
        const int r = q + 8 * i, n = min(n0 + r % OUT, a.N - 1);            // (behind the last row: the last row again, not stored)
        w[i] = W + (int64_t)(DUAL && r >= OUT ? a.N + n : n) * a.ldw;
    }
    const uint4 zero = make_uint4(0, 0, 0, 0);
    uint4 wv[WR][U][V];
    auto fetch = [&](int s) {
#pragma unroll
        for (int u = 0; u < U; ++u)
#pragma unroll
            for (int i = 0; i < WR; ++i) {
                const int k = (s + u) * 32 * V + k8;
#pragma unroll
                for (int e = 0; e < V; ++e) wv[i][u][e] = zero;
                if (k < a.K) load_weights<V>(wv[i][u], w[i] + k);           // (K is a multiple of 8 V)
            }
    };
    // (a model's weights: on their way while the kernel in front of this one ends.  Not where experts without rows are left out)
    const bool early = a.weights_ready && a.grp_off == nullptr;
    if (early) fetch(warp * U);
    chain_wait();
    int row_lo = 0, rows = a.M;
    if (a.grp_off != nullptr) { row_lo = a.grp_off[g]; rows = a.grp_off[g + 1] - row_lo; }
    if (rows <= 0) return;
#pragma unroll
    for (int i = 0; i < NT; ++i) {
        const int m = q + 8 * i;
        x[i] = m < rows ? A + (int64_t)(a.row_src ? a.row_src[row_lo + m] : row_lo + m) * a.lda : nullptr;
    }
    if (!early) fetch(warp * U);
    float sum[R == 16 ? NT : 1][4] = {};
    for (int s = warp * U; s * 32 * V < a.K; s += KW * U) {
        uint4 xv[NT][U][V];
        if (s != warp * U) fetch(s);
#pragma unroll
        for (int u = 0; u < U; ++u)
#pragma unroll
            for (int i = 0; i < NT; ++i) {
                const int k = (s + u) * 32 * V + k8;
#pragma unroll
                for (int e = 0; e < V; ++e) xv[i][u][e] = zero;
                if (x[i] != nullptr && k < a.K) load_rows<V>(xv[i][u], x[i] + k);
            }
#pragma unroll
        for (int i = 0; i < (R == 16 ? NT : 1); ++i) {
            float d[2 * U * V][4] = {};
#pragma unroll
            for (int u = 0; u < U; ++u)
#pragma unroll
                for (int e = 0; e < V; ++e) {
                    float (&d0)[4] = d[2 * (u * V + e)], (&d1)[4] = d[2 * (u * V + e) + 1];
                    const uint4 xl = xv[i][u][e], w0 = wv[0][u][e];
                    if constexpr (R == 16) {
                        const uint4 w1 = wv[WR - 1][u][e];
                        mma_16816(d0, w0.x, w1.x, w0.y, w1.y, xl.x, xl.y);
                        mma_16816(d1, w0.z, w1.z, w0.w, w1.w, xl.z, xl.w);
                    } else {
                        const uint4 xh = NT == 2 ? xv[NT - 1][u][e] : zero;
                        mma_16816(d0, xl.x, xh.x, xl.y, xh.y, w0.x, w0.y);
                        mma_16816(d1, xl.z, xh.z, xl.w, xh.w, w0.z, w0.w);
                    }
                }
#pragma unroll
            for (int h = U * V; h > 0; h >>= 1)
#pragma unroll
                for (int c = 0; c < h; ++c)
#pragma unroll
                    for (int e = 0; e < 4; ++e) d[c][e] += d[c + h][e];
#pragma unroll
            for (int e = 0; e < 4; ++e) sum[i][e] += d[0][e];
        }
    }
#pragma unroll
    for (int i = 0; i < (R == 16 ? NT : 1); ++i)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int lo = (lane & 3) * 2 + (e & 1), hi = q + (e >> 1) * 8;
            if (R == 16) part[warp][i * 8 + lo][hi] = sum[i][e];
            else if (hi < NT * 8) part[warp][hi][lo] = sum[i][e];
        }
    __syncthreads();
    TC* C = (TC*)a.C + (int64_t)g * a.c_goff;
    for (int i = threadIdx.x; i < OUT * NT * 8; i += 32 * KW) {
        const int m = i / OUT, o = i % OUT, n = n0 + o;
        if (n >= a.N || m >= rows) continue;
        double s[4] = {}, s2[4] = {};
#pragma unroll
        for (int p = 0; p < KW; ++p) {
            s[p & 3] += (double)part[p][m][o];
            if (DUAL) s2[p & 3] += (double)part[p][m][o + OUT];
        }
        const int64_t row = row_lo + m;
        C[row * a.ldc + n] = from_f32<TC>(finish<DUAL>(a, (float)((s[0] + s[1]) + (s[2] + s[3])), (float)((s2[0] + s2[1]) + (s2[2] + s2[3])), g, row, n));
    }
}

// The weight's sizes (and V) choose the order of the sums: warps that share a tile's k so that each has all or half of its pieces in flight at
// once, up to what the SMs hold.  Tiles of 8 weight rows (the activations are the 16-row operand then) where tiles of 16 would leave SMs
// idle, and for 9 to 16 activation rows, whose pieces the registers hold beside one weight row's; the sums are the same in both.
// us, weights of 50 to 200 MB in turn, 8 rows, the best of the others / the chosen one: 1024 x 1024 2.4 / 2.5, 2048 x 1024 2.6 / 2.6,
// 8192 x 1024 5.3 / 5.5, 1024 x 2048 2.9 / 2.7, 6144 x 2048 7.3 / 6.7, 1024 x 4096 5.2 / 5.0, 3088 x 4096 9.2 / 7.9.
template <typename TC, bool DUAL, int NT, int KW, int U, int V>
static void launch_skinny_tiles(const GemmArgs& a, int groups, int64_t tiles, cudaStream_t st) {
    if (NT == 1 && tiles >= 128) chain_launch(gemm_skinny_kernel<TC, DUAL, 16, 1, KW, U, V>, dim3((a.N + (DUAL ? 7 : 15)) / (DUAL ? 8 : 16), groups), 32 * KW, 0, st, a);
    else chain_launch(gemm_skinny_kernel<TC, DUAL, 8, NT, KW, U, V>, dim3((a.N + (DUAL ? 3 : 7)) / (DUAL ? 4 : 8), groups), 32 * KW, 0, st, a);
}
template <typename TC, bool DUAL, int NT, int V>
static void launch_skinny_rows(const GemmArgs& a, int groups, cudaStream_t st) {
    const int64_t tiles = (int64_t)((a.N + (DUAL ? 7 : 15)) / (DUAL ? 8 : 16)) * groups;
    constexpr int U = 2 / V;                                // steps of 64 k
    if (a.K <= 512 || (a.K <= 1024 && tiles >= 400)) launch_skinny_tiles<TC, DUAL, NT, 8, U, V>(a, groups, tiles, st);
    else if (a.K <= 1024 || tiles > 200) launch_skinny_tiles<TC, DUAL, NT, 8, 2 * U, V>(a, groups, tiles, st);
    else if (tiles > 100) launch_skinny_tiles<TC, DUAL, NT, 16, U, V>(a, groups, tiles, st);
    else launch_skinny_tiles<TC, DUAL, NT, 16, 2 * U, V>(a, groups, tiles, st);
}
template <typename TC, int V>
static void launch_skinny_pieces(const GemmArgs& a, int groups, bool dual, cudaStream_t st) {
    if (dual) a.M <= 8 ? launch_skinny_rows<TC, true, 1, V>(a, groups, st) : launch_skinny_rows<TC, true, 2, V>(a, groups, st);
    else a.M <= 8 ? launch_skinny_rows<TC, false, 1, V>(a, groups, st) : launch_skinny_rows<TC, false, 2, V>(a, groups, st);
}
// 32-byte pieces where every row of both operands starts on such a boundary: a load then takes whole lines of eight rows, not halves
// (2048 x 1024 2.9 -> 2.6, 1024 x 2048 3.7 -> 2.7).
template <typename TC>
static void launch_skinny(const GemmArgs& a, int groups, bool dual, cudaStream_t st) {
    const bool wide = a.K % 16 == 0 && a.lda % 16 == 0 && a.ldw % 16 == 0 && a.a_goff % 16 == 0 && a.w_gstride % 16 == 0 &&
                      (((uintptr_t)a.A | (uintptr_t)a.W) & 31) == 0;
    if (wide) launch_skinny_pieces<TC, 2>(a, groups, dual, st);
    else launch_skinny_pieces<TC, 1>(a, groups, dual, st);
}

// Few rows of 32-bit operands, on the multiply-add pipe.  What it waits for is the latency of a
// row's loads, one after the other, so a weight row is split over KW warps (k in pieces of 16 bytes a lane, warp after
// warp), a thread takes four weight rows (with DUAL: the gate and up rows of two outputs) and has the 16-byte loads of two
// of its pieces in flight; a block of four warps covers 4 / KW such sets of rows.  Sums are kept as even and odd halves (one
// instruction for both), added over the lanes by a tree that hands every lane fewer values at each level, then over the
// warps in order: the order depends on K alone, so a row's result does not depend on the other rows.
constexpr int SK_ROWS = 4, SK_WARPS = 4;

__device__ __forceinline__ void unpack_piece(const uint4& v, f32x2 (&f)[2]) {
    f[0] = (f32x2)v.y << 32 | v.x;
    f[1] = (f32x2)v.w << 32 | v.z;
}

template <bool DUAL, int MT, int KW>
__global__ void __launch_bounds__(32 * SK_WARPS) gemm_rows_kernel(GemmArgs a) {
    constexpr int OUTS = DUAL ? SK_ROWS / 2 : SK_ROWS, SETS = SK_WARPS / KW, V = SK_ROWS * MT;      // outputs per set; sums per thread
    constexpr int PV = 4, STEP = KW * 32 * PV;              // numbers of a piece; k of the warps' pieces together
    __shared__ float part[SK_WARPS][V];
    chain_wait();
    const int g = blockIdx.z;
    int row_lo = 0, rows = a.M;
    if (a.grp_off != nullptr) { row_lo = a.grp_off[g]; rows = a.grp_off[g + 1] - row_lo; }
    const int m0 = blockIdx.y * MT;
    if (m0 >= rows) return;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, set = warp / KW, kw = warp % KW;
    const int n0 = (blockIdx.x * SETS + set) * OUTS;
    const float* A = (const float*)a.A + (int64_t)g * a.a_goff;
    const float* W = (const float*)a.W + (int64_t)g * a.w_gstride;
    const float* wrow[SK_ROWS];
#pragma unroll
    for (int i = 0; i < SK_ROWS; ++i) {
        const int n = min(DUAL ? (n0 + (i >> 1)) : (n0 + i), a.N - 1);      // behind the last row: the last row again, not stored
        wrow[i] = W + (int64_t)(DUAL ? ((i & 1) * a.N + n) : n) * a.ldw;
    }
    const float* arow[MT];
#pragma unroll
    for (int m = 0; m < MT; ++m) {
        const int p = row_lo + min(m0 + m, rows - 1);
        arow[m] = A + (int64_t)(a.row_src ? a.row_src[p] : p) * a.lda;
    }
    f32x2 acc[SK_ROWS][MT];
#pragma unroll
    for (int i = 0; i < SK_ROWS; ++i)
#pragma unroll
        for (int m = 0; m < MT; ++m) acc[i][m] = 0ull;
    const uint4 zero = make_uint4(0, 0, 0, 0);
    for (int k = (kw * 32 + lane) * PV; k < a.K; k += 2 * STEP) {
        const int k2 = k + STEP;
        uint4 wv[2][SK_ROWS];
#pragma unroll
        for (int i = 0; i < SK_ROWS; ++i) wv[0][i] = __ldg(reinterpret_cast<const uint4*>(wrow[i] + k));
#pragma unroll
        for (int i = 0; i < SK_ROWS; ++i) wv[1][i] = k2 < a.K ? __ldg(reinterpret_cast<const uint4*>(wrow[i] + k2)) : zero;
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            f32x2 wf[SK_ROWS][PV / 2];
#pragma unroll
            for (int i = 0; i < SK_ROWS; ++i) unpack_piece(wv[u][i], wf[i]);
#pragma unroll
            for (int m = 0; m < MT; ++m) {
                f32x2 af[PV / 2];
                unpack_piece(u == 0 || k2 < a.K ? *reinterpret_cast<const uint4*>(arow[m] + (u ? k2 : k)) : zero, af);
#pragma unroll
                for (int i = 0; i < SK_ROWS; ++i)
#pragma unroll
                    for (int e = 0; e < PV / 2; ++e) acc[i][m] = fma2(af[e], wf[i][e], acc[i][m]);
            }
        }
    }
    float v[V];
#pragma unroll
    for (int i = 0; i < SK_ROWS; ++i)
#pragma unroll
        for (int m = 0; m < MT; ++m) {
            const float2 h = unpack2(acc[i][m]);
            v[i * MT + m] = h.x + h.y;
        }
    // the lanes' sums: a lane keeps half of its values at each level while it has several
#pragma unroll
    for (int o = 16, c = V; o > 0; o >>= 1) {
        if (c > 1) {
            c >>= 1;
#pragma unroll
            for (int i = 0; i < V / 2; ++i) {
                if (i >= c) continue;
                const float send = (lane & o) ? v[i] : v[i + c], keep = (lane & o) ? v[i + c] : v[i];
                v[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
            }
        } else {
            v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
        }
    }
    constexpr int per = 32 / V;                                             // lanes that hold the same value
    if (lane % per == 0) part[warp][lane / per] = v[0];
    __syncthreads();
    float* C = (float*)a.C + (int64_t)g * a.c_goff;
    for (int i = threadIdx.x; i < SETS * OUTS * MT; i += 32 * SK_WARPS) {
        const int st = i / (OUTS * MT), o = i % (OUTS * MT) / MT, m = i % MT, n = (blockIdx.x * SETS + st) * OUTS + o;
        if (n >= a.N || m0 + m >= rows) continue;
        float s = 0.f, s2 = 0.f;
#pragma unroll
        for (int q = 0; q < KW; ++q) {
            s += part[st * KW + q][(DUAL ? 2 * o : o) * MT + m];
            if (DUAL) s2 += part[st * KW + q][(2 * o + 1) * MT + m];
        }
        const int64_t row = row_lo + m0 + m;
        C[row * a.ldc + n] = finish<DUAL>(a, s, s2, g, row, n);
    }
}

// K alone chooses how many warps share a row: with one the loop over k is the critical path from 64 pieces on.
static void launch_rows(const GemmArgs& a, int groups, bool dual, cudaStream_t st) {
    const int pieces = a.K / 4, kw = pieces >= 128 ? 4 : (pieces >= 64 ? 2 : 1);
    const int outs_per_block = SK_WARPS / kw * (dual ? SK_ROWS / 2 : SK_ROWS);
    const int mt = a.M <= 1 ? 1 : (a.M <= 2 ? 2 : (a.M <= 4 ? 4 : 8));
    const dim3 grid((a.N + outs_per_block - 1) / outs_per_block, (a.M + mt - 1) / mt, groups), block(32 * SK_WARPS);
#define UMBS_SK2(MT, KW)                                                                  \
    do {                                                                                  \
        if (dual) chain_launch(gemm_rows_kernel<true, MT, KW>, grid, block, 0, st, a);    \
        else chain_launch(gemm_rows_kernel<false, MT, KW>, grid, block, 0, st, a);        \
    } while (0)
#define UMBS_SK(MT)                                                                   \
    do {                                                                              \
        if (kw == 4) UMBS_SK2(MT, 4);                                                 \
        else if (kw == 2) UMBS_SK2(MT, 2);                                            \
        else UMBS_SK2(MT, 1);                                                         \
    } while (0)
    if (mt == 1) UMBS_SK(1);
    else if (mt == 2) UMBS_SK(2);
    else if (mt == 4) UMBS_SK(4);
    else UMBS_SK(8);
#undef UMBS_SK
#undef UMBS_SK2
}

template <typename TA, typename TC, int RT>
static void launch_simt_rows(const GemmArgs& a, int groups, bool dual, cudaStream_t st) {
    const int out = dual ? BN / 2 : BN;
    const dim3 grid((a.N + out - 1) / out, (a.M + 8 * RT - 1) / (8 * RT), groups);
    const bool vec = a.lda % 4 == 0 && a.ldw % 4 == 0 && a.a_goff % 4 == 0 && a.w_gstride % 4 == 0 && (((uintptr_t)a.A | (uintptr_t)a.W) & 15) == 0;
    const bool vec_c = a.ldc % 4 == 0 && a.c_goff % 4 == 0 && ((uintptr_t)a.C & 15) == 0;
    if (dual) gemm_simt_kernel<TA, TC, true, RT><<<grid, 64, 0, st>>>(a, vec, vec_c);
    else gemm_simt_kernel<TA, TC, false, RT><<<grid, 64, 0, st>>>(a, vec, vec_c);
}
// Tiles of 64 rows where they give every SM a block, else of 16: with few blocks a tile's own length counts, whether its rows are
// there or not (us with 4 x 4 outputs a thread over 256 threads, as before the 8 x 8 tiles / 64 rows / 16 rows; K = 1024: 1 row to
// 3088 columns 71 / 74 / 47, 64 rows to 1024 columns 82 / 85 / 45, 64 rows of 16 groups, K = 64: 11 / 29 / 9; 100 rows to 8192
// columns, 256 blocks: 109 / 89 / 114).
template <typename TA, typename TC>
static void launch_simt(const GemmArgs& a, int groups, bool dual, cudaStream_t st) {
    const int out = dual ? BN / 2 : BN;
    if ((int64_t)((a.N + out - 1) / out) * ((a.M + 63) / 64) * groups < 148) launch_simt_rows<TA, TC, 2>(a, groups, dual, st);
    else launch_simt_rows<TA, TC, 8>(a, groups, dual, st);
}

}  // namespace umbs

using namespace umbs;

static int gemm_run(int dtype, const void* A, int64_t lda, int a_goff, const void* W, int64_t ldw, int64_t w_gstride,
                    void* C, int64_t ldc, int c_goff, int c_f32, int M, int N, int K, int groups,
                    const int32_t* grp_off, const int32_t* row_src, int dual, float limit, const float* bias,
                    const float* out_gate, int64_t ld_gate, int gate_goff, int gate_n, int unary, float p0, float p1, int unary_cols,
                    umbs_stream_t stream, int rows_total = 0);

extern "C" int umbs_gemm(int dtype, const void* A, int64_t lda, int a_goff, const void* W, int64_t ldw, int64_t w_gstride,
                         void* C, int64_t ldc, int c_goff, int c_f32, int M, int N, int K, int groups,
                         const int32_t* grp_off, const int32_t* row_src, int dual, float limit, umbs_stream_t stream) {
    return umbs_gemm_ex(dtype, A, lda, a_goff, W, ldw, w_gstride, C, ldc, c_goff, c_f32, M, N, K, groups, grp_off, row_src, dual,
                        limit, nullptr, nullptr, 0, 0, stream);
}

extern "C" int umbs_gemm_sorted(int dtype, const void* A, int64_t lda, const void* W, int64_t ldw, int64_t w_gstride, void* C, int64_t ldc,
                                int c_f32, int M, int rows, int N, int K, int groups, const int32_t* grp_off, const int32_t* row_src, int dual,
                                float limit, umbs_stream_t stream) {
    if (rows <= 0 || N <= 0) return 0;
    if (C == nullptr || grp_off == nullptr || ldc < N) return UMB_ERR_ARG;
    return gemm_run(dtype, A, lda, 0, W, ldw, w_gstride, C, ldc, 0, c_f32, M, N, K, groups, grp_off, row_src, dual, limit, nullptr, nullptr, 0, 0,
                    1, 0, 0.f, 0.f, 0, stream, rows);
}

extern "C" int umbs_gemm_ex(int dtype, const void* A, int64_t lda, int a_goff, const void* W, int64_t ldw, int64_t w_gstride,
                            void* C, int64_t ldc, int c_goff, int c_f32, int M, int N, int K, int groups,
                            const int32_t* grp_off, const int32_t* row_src, int dual, float limit, const float* bias,
                            const float* out_gate, int64_t ld_gate, int gate_goff, umbs_stream_t stream) {
    return gemm_run(dtype, A, lda, a_goff, W, ldw, w_gstride, C, ldc, c_goff, c_f32, M, N, K, groups, grp_off, row_src, dual, limit,
                    bias, out_gate, ld_gate, gate_goff, 1, 0, 0.f, 0.f, 0, stream);
}

extern "C" int umbs_gemm_unary(int dtype, const void* A, int64_t lda, int a_goff, const void* W, int64_t ldw, int64_t w_gstride,
                               void* C, int64_t ldc, int c_goff, int c_f32, int M, int N, int K, int groups, const float* bias,
                               int unary, float p0, float p1, umbs_stream_t stream) {
    return umbs_gemm_unary_cols(dtype, A, lda, a_goff, W, ldw, w_gstride, C, ldc, c_goff, c_f32, M, N, K, groups, bias, unary, p0, p1,
                                0, stream);
}

extern "C" int umbs_gemm_unary_cols(int dtype, const void* A, int64_t lda, int a_goff, const void* W, int64_t ldw, int64_t w_gstride,
                                    void* C, int64_t ldc, int c_goff, int c_f32, int M, int N, int K, int groups, const float* bias,
                                    int unary, float p0, float p1, int unary_cols, umbs_stream_t stream) {
    if (unary < 0 || unary > UMBS_UNARY_SCALE || unary_cols < 0) return UMB_ERR_ARG;
    return gemm_run(dtype, A, lda, a_goff, W, ldw, w_gstride, C, ldc, c_goff, c_f32, M, N, K, groups, nullptr, nullptr, 0, 0.f, bias,
                    nullptr, 0, 0, 1, unary, p0, p1, unary_cols > 0 ? unary_cols : N, stream);
}

extern "C" int umbs_gemm_head_gate(int dtype, const void* A, int64_t lda, int a_goff, const void* W, int64_t ldw, int64_t w_gstride,
                                   void* C, int64_t ldc, int c_goff, int c_f32, int M, int N, int K, int groups, const float* out_gate,
                                   int64_t ld_gate, umbs_stream_t stream) {
    return gemm_run(dtype, A, lda, a_goff, W, ldw, w_gstride, C, ldc, c_goff, c_f32, M, N, K, groups, nullptr, nullptr, 0, 0.f, nullptr,
                    out_gate, ld_gate, 1, 0, 0, 0.f, 0.f, 0, stream);
}

constexpr int kFewRows = 16;
// Streamed fp32 rows take 2 us and one for 6.5 million products, tiles on the tensor core 6 us and 1.3 for each 64 of k.  (us, multiply-add
// tiles / streamed / tensor core, K = 1024: one row of 3088 columns 54 / 4.6 / 29, 64 rows of 1024 45 / 12 / 25, of 3088 51 / 32 / 28, of
// 8192 73 / 78 / 31; 200 rows of 3088 85 / - / 32; 128 rows, K = 4096, to 1024 columns 184 / 60 / 90.)
// (the streamed rows are the grid's second extent)
static bool f32_streams(int M, int64_t w_rows, int K, int groups) {
    return M <= 4096 && (M <= kFewRows || (double)M * w_rows * groups * K <= 8.5e6 * (K / 64 + 4));
}

extern "C" int umbs_gemm_kernel(int dtype, int M, int N, int K, int groups, int sorted, int dual, int sms) {
    if (M <= 0 || N <= 0 || K <= 0 || groups <= 0 || sms <= 0) return UMB_ERR_ARG;
    if (dtype == UMBS_F32) return K % 4 ? UMBS_GEMM_GENERAL : f32_streams(M, (int64_t)N * (dual ? 2 : 1), K, groups) ? UMBS_GEMM_FEW_ROWS : UMBS_GEMM_SPLIT;
    if (dtype != UMBS_BF16) return UMB_ERR_ARG;
    if (K % 8 == 0 && M <= kFewRows) return UMBS_GEMM_FEW_ROWS;
    return K % 32 ? UMBS_GEMM_GENERAL : tc_tile_columns(M, N, K, groups, dual != 0, sorted != 0, sorted != 0, sms);
}

static int gemm_run(int dtype, const void* A, int64_t lda, int a_goff, const void* W, int64_t ldw, int64_t w_gstride,
                    void* C, int64_t ldc, int c_goff, int c_f32, int M, int N, int K, int groups,
                    const int32_t* grp_off, const int32_t* row_src, int dual, float limit, const float* bias,
                    const float* out_gate, int64_t ld_gate, int gate_goff, int gate_n, int unary, float p0, float p1, int unary_cols,
                    umbs_stream_t stream, int rows_total) {
    cudaStream_t st = (cudaStream_t)stream;
    // (the tensor-core tiles take every row of every group and clear what is left themselves: two products of a prompt's 8192 sorted
    // rows, 18 us of clearing first)
    auto clear = [&]() -> cudaError_t {
        const size_t es = dtype == UMBS_F32 || c_f32 ? 4 : 2;
        return rows_total > 0 ? cudaMemset2DAsync(C, ldc * es, 0, N * es, rows_total, st) : cudaSuccess;
    };
    if (M <= 0 || N <= 0 || groups <= 0) return (int)clear();
    if (K <= 0 || A == nullptr || W == nullptr || C == nullptr) return UMB_ERR_ARG;
    GemmArgs a{A, lda, a_goff, W, ldw, w_gstride, C, ldc, c_goff, M, N, K, grp_off, row_src, limit,
               (dual == UMBS_ACT_GELU_TANH || dual == UMBS_ACT_SILU) ? dual : UMBS_ACT_CLAMPED_GLU,
               bias, out_gate, ld_gate, gate_goff, gate_n, unary, p0, p1, unary_cols, rows_total,
               in_chain()};                                 // (a model's products: W is a layer's weight)
    if (dtype == UMBS_F32) {                                              // activations are fp32 too: c_f32 changes nothing
        if (const cudaError_t e = clear()) return (int)e;
        const bool vec = (K % 4 == 0) && (lda % 4 == 0) && (ldw % 4 == 0) && (a_goff % 4 == 0) && (w_gstride % 4 == 0) &&
                         ((uintptr_t)A % 16 == 0) && ((uintptr_t)W % 16 == 0);
        // (the tiles count rows in 16-byte pieces of 32 bits: strides forwards, 16 GB of dense rows and of weights)
        const int64_t w_rows = (int64_t)N * (dual ? 2 : 1);
        const bool split = vec && lda >= 0 && ldw >= 0 && lda <= UINT32_MAX / std::max(M, 1) && ldw <= UINT32_MAX / w_rows;
        if (vec && f32_streams(M, w_rows, K, groups)) {
            launch_rows(a, groups, dual != 0, st);
        } else if (split) {
            const int rc = launch_gemm_split(a, groups, dual != 0, st);
            if (rc != 0) return rc;
        } else {
            launch_simt<float, float>(a, groups, dual != 0, st);
        }
    } else if (dtype == UMBS_BF16) {
        // 16-byte loads: every row start and group offset must sit on a 16-byte boundary
        const bool vec = (K % 8 == 0) && (lda % 8 == 0) && (ldw % 8 == 0) && (a_goff % 8 == 0) && (w_gstride % 8 == 0) &&
                         ((uintptr_t)A % 16 == 0) && ((uintptr_t)W % 16 == 0);
        // (rows that overlap, one row repeated among them: not described by a tensor map, they take the general kernel)
        const bool tc = vec && (K % 32 == 0) && lda >= K && ldw >= K;
        if (vec && M <= kFewRows) {
            if (const cudaError_t e = clear()) return (int)e;
            if (c_f32) launch_skinny<float>(a, groups, dual != 0, st);
            else launch_skinny<__nv_bfloat16>(a, groups, dual != 0, st);
        } else {
            const int rc = tc ? launch_gemm_tc(a, groups, dual != 0, c_f32 != 0, st) : UMB_ERR_DRIVER;
            if (rc == UMB_ERR_DRIVER) {
                if (const cudaError_t e = clear()) return (int)e;         // (also strides that no tensor map describes: groups that run backwards)
                if (c_f32) launch_simt<__nv_bfloat16, float>(a, groups, dual != 0, st);
                else launch_simt<__nv_bfloat16, __nv_bfloat16>(a, groups, dual != 0, st);
            } else if (rc != 0) {
                return rc;
            }
        }
    } else {
        return UMB_ERR_ARG;
    }
    count_launches(1);
    return (int)cudaGetLastError();
}
