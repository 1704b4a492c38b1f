// What the AWQ product kernels share: the packed record, the stream-K schedule, the dequantisation of a word, the parameters and the
// epilogues of 16 token columns (gemm.cu, gemm_wide.cu).
#pragma once
#include <cuda.h>

#include "common.cuh"
#include "internal.h"

namespace umb {

constexpr int kTileN = 128;              // output features per tile (UMMA M)
constexpr int kGroup = 128;              // AWQ group size == k per AWQ unit
constexpr int kRecordBytes = 8512;       // 8192 nibble bytes + 256 scale bytes + 64 zero bytes (what a TMA copy moves)
#ifndef UMB_RECORD_STRIDE
#define UMB_RECORD_STRIDE 8512
#endif
constexpr int kRecordStride = UMB_RECORD_STRIDE;   // distance between records in the stream
constexpr int kRecScaleOff = 8192;
constexpr int kRecZeroOff = 8448;
// nibble position of the i-th of 8 consecutive values inside a 32-bit word: (0,4,1,5,2,6,3,7).
// Used by the AutoAWQ checkpoint layout (along N) and by our repacked stream (along K): nibbles p
// and p + 4 hold consecutive values, so (w >> 4p) & 0x000f000f yields an ordered pair.
__host__ __device__ __forceinline__ int nib_pos(int i) { return (i >> 1) + ((i & 1) << 2); }

// ------------------------------------------------------------------------------------------------
// stream-K schedule helpers
// ------------------------------------------------------------------------------------------------
__device__ __forceinline__ long long sk_begin(long long c, long long U, long long P) { return c * U / P; }
__device__ __forceinline__ int sk_owner(long long u, long long U, long long P) {
    long long c = u * P / U;
    while (c + 1 < P && sk_begin(c + 1, U, P) <= u) ++c;
    while (c > 0 && sk_begin(c, U, P) > u) --c;
    return (int)c;
}

// One 32-bit word of the packed stream = 8 consecutive k of one feature row, nibble i at position
// (0,4,1,5,2,6,3,7)[i].  Nibbles p and p+4 are extracted together as an fp16 pair:
//   p = 0: (w      & 0x000f000f) | 0x6400 = 1024 +    q      p = 1: (w      & 0x00f000f0) | 0x6400 = 1024 + 16 q
//   p = 2: (w >> 8 & 0x000f000f) | 0x6400                     p = 3: (w >> 8 & 0x00f000f0) | 0x6400
// then   even: (1024 + q) - (1024 + z)        odd: (1024 + 16 q) * (1/16) - (64 + z)
// are both EXACT (q - z), and one multiply by the group scale rounds once: fp16((q - z) * s).
template <uint32_t kMask>
__device__ __forceinline__ uint32_t lop3_and_or(uint32_t a, uint32_t c) {
    uint32_t d;
    asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(d) : "r"(a), "n"(kMask), "r"(c));
    return d;
}
__device__ __forceinline__ __half2 as_h2(uint32_t v) { return *reinterpret_cast<__half2*>(&v); }
__device__ __forceinline__ uint32_t as_u32(__half2 v) { return *reinterpret_cast<uint32_t*>(&v); }
__device__ __forceinline__ void dequant_word(uint32_t w, uint32_t magic, __half2 ce, __half2 neg_co, __half2 s2,
                                             uint32_t* out) {
    const __half2 sixteenth = as_h2(0x2C002C00u);                 // 1/16
    const uint32_t w8 = w >> 8;
    // (t - ce) and fma(t, 1/16, -co) are exact; the multiply by the scale is the single rounding
    out[0] = as_u32(__hmul2(__hsub2(as_h2(lop3_and_or<0x000f000fu>(w, magic)), ce), s2));
    out[1] = as_u32(__hmul2(__hfma2(as_h2(lop3_and_or<0x00f000f0u>(w, magic)), sixteenth, neg_co), s2));
    out[2] = as_u32(__hmul2(__hsub2(as_h2(lop3_and_or<0x000f000fu>(w8, magic)), ce), s2));
    out[3] = as_u32(__hmul2(__hfma2(as_h2(lop3_and_or<0x00f000f0u>(w8, magic)), sixteenth, neg_co), s2));
}
__device__ __forceinline__ uint4 lds128(uint32_t addr) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr));
    return v;
}
__device__ __forceinline__ uint32_t lds32(uint32_t addr) {
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(addr));
    return v;
}
__device__ __forceinline__ uint32_t lds16(uint32_t addr) {
    unsigned short v;
    asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(addr));
    return v;
}

struct GemmParams {
    const unsigned char* packed;   // AWQ stream (kAwq) -- else unused
    int M, K, N_total;             // N_total = output features (rows of W)
    int units_per_tile;            // K / 128 (AWQ) or K / 64 (fp16)
    int tiles;
    void* y;
    int64_t ldy;
    int mode;
    const __half* bias;
    const __half* residual;
    int64_t ld_residual;
    int vec_ok;                    // y (and the residual) can be accessed with 16-byte vectors
    int rope_vec_ok;               // same for q_out / k_cache / v_cache / cos / sin of UMB_EPI_ROPE_QKV
    unsigned long long* argmax;
    int* counters;                 // [tiles]
    float* slots;                  // [tiles + grid][MPAD][128]
    umb_rope_epilogue_t rope;      // UMB_EPI_ROPE_QKV operands (by value)
    int stages;                    // depth of the shared-memory ring
    unsigned long long* trace;     // debug timeline [grid][16] (UMB_GEMM_TRACE=1), else NULL
};

__device__ __forceinline__ float silu_f(float f) { return f / (1.f + expf(-f)); }
__device__ __forceinline__ unsigned int orderable_f32_g(float f) {
    const unsigned int u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

// Epilogue of 16 token columns [m0, m0 + 16) for feature lane `fl` (0..127) of tile `tile`.  The four warps that run it
// share the staging rows `exch` and the named barrier `bar`.
__device__ __forceinline__ void epilogue_chunk(const GemmParams& p, int tile, int fl, int m0, const float (&v)[16],
                                               __half* exch, uint32_t bar = 2) {
    const int n = tile * kTileN + fl;
    if (p.mode == UMB_EPI_SILU_MUL) {
        // lanes 0..63 hold `gate`, lanes 64..127 `up` of output features tile*64 + (fl & 63).  Both halves of the
        // 16-row chunk are staged as fp16 (the rounding point of the reference's gate / up tensors), every thread
        // then finishes 8 of the 16 x 64 outputs in place, and the tile leaves with one 16-byte store per thread.
        __half* g_t = exch;                    // [16][64] gate, overwritten by the outputs
        __half* u_t = exch + 16 * 64;          // [16][64] up
        {
            __half* dst = (fl < 64 ? g_t : u_t) + (fl & 63);
#pragma unroll
            for (int j = 0; j < 16; ++j) dst[j * 64] = __float2half_rn(v[j]);
        }
        named_bar_sync(bar, 128);
        {
            const int col = fl & 63, r0 = fl >> 6;
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const int r = r0 + 2 * i;
                const __half g = g_t[r * 64 + col];
                const __half sl = __float2half_rn(silu_f(__half2float(g)));
                g_t[r * 64 + col] = __hmul(sl, u_t[r * 64 + col]);
            }
        }
        named_bar_sync(bar, 128);
        {
            const int row = fl >> 3, seg = (fl & 7) * 8;
            const int no = tile * 64 + seg;
            if (row < p.M - m0 && no + 8 <= p.N_total / 2) {
                __half* yp = reinterpret_cast<__half*>(p.y) + (int64_t)(m0 + row) * p.ldy + no;
                if (p.vec_ok) {
                    *reinterpret_cast<uint4*>(yp) = *reinterpret_cast<const uint4*>(g_t + row * 64 + seg);
                } else {
#pragma unroll
                    for (int c = 0; c < 8; ++c) yp[c] = g_t[row * 64 + seg + c];
                }
            }
        }
        named_bar_sync(bar, 128);
        return;
    }
    if (p.mode == UMB_EPI_ROPE_QKV) {
        // q|k|v projection with RoPE + KV append fused: the rotation partner of feature d is d +- D/2, i.e. lane
        // fl ^ (D/2) of the same tile (128 % D == 0); the pair is exchanged through shared memory as fp16 -- the
        // rounding point where the reference holds the fp16 q / k / v tensors.
        const umb_rope_epilogue_t& r = p.rope;
        const int D = r.head_dim, half_d = D >> 1;
        const bool n_ok = n < p.N_total;
        __half h[16];
        const bool has_bias = p.bias != nullptr && n_ok;
        const __half qb = has_bias ? p.bias[n] : __float2half_rn(0.f);
#pragma unroll
        for (int j = 0; j < 16; ++j) {
            h[j] = __float2half_rn(v[j]);
            if (has_bias) h[j] = __hadd(h[j], qb);
            exch[j * kTileN + fl] = h[j];
        }
        const int base = r.n_dev ? r.n_dev[0] : 0;
        const int mcols = p.M - m0;
        if (p.rope_vec_ok) {
            // Staged form: the cos / sin rows of the chunk's 16 positions are fetched with 16-byte loads by the whole
            // group (two dependent round trips in total instead of three per token through one register), the
            // rotated tile is finished in shared memory and leaves with two 16-byte stores per thread.
            __half* cos_t = exch + 16 * kTileN;          // [16][D]
            __half* sin_t = cos_t + 16 * kTileN;         // [16][D]
            const int segs = D >> 3;                     // 16-byte segments per table row
            const int64_t* pid = r.position_ids + (r.n_dev ? base + r.row_offset : 0) + m0;
#pragma unroll
            for (int it = 0; it < 2; ++it) {
                const int sidx = fl + it * 128;
                const int row = sidx / segs, seg = sidx - row * segs;
                if (sidx < 16 * segs && row < mcols) {
                    const int64_t off = pid[row] * D + seg * 8;
                    *reinterpret_cast<uint4*>(cos_t + row * D + seg * 8) =
                        *reinterpret_cast<const uint4*>(reinterpret_cast<const __half*>(r.cos) + off);
                    *reinterpret_cast<uint4*>(sin_t + row * D + seg * 8) =
                        *reinterpret_cast<const uint4*>(reinterpret_cast<const __half*>(r.sin) + off);
                }
            }
            named_bar_sync(bar, 128);
            const int head = n / D, d = n - head * D;
            const bool rot = n_ok && head < r.num_q_heads + r.num_kv_heads;
            __half o[16];
#pragma unroll
            for (int j = 0; j < 16; ++j) {
                o[j] = h[j];
                if (rot && j < mcols) {
                    const __half pr = exch[j * kTileN + (fl ^ half_d)];
                    // (x * cos) + (rotate_half(x) * sin): two products and one sum, each rounded (no fma)
                    o[j] = __hadd_rn(__hmul_rn(h[j], cos_t[j * D + d]), __hmul_rn(d < half_d ? __hneg(pr) : pr, sin_t[j * D + d]));
                }
            }
            named_bar_sync(bar, 128);                  // every partner value has been read
#pragma unroll
            for (int j = 0; j < 16; ++j) exch[j * kTileN + fl] = o[j];
            named_bar_sync(bar, 128);
#pragma unroll
            for (int it = 0; it < 2; ++it) {
                const int sidx = fl + it * 128, row = sidx >> 4, c0 = (sidx & 15) * 8;
                const int n0 = tile * kTileN + c0;
                if (row < mcols && n0 + 8 <= p.N_total) {
                    const int hd = n0 / D, d0 = n0 - hd * D, m = m0 + row;
                    __half* dst;
                    if (hd < r.num_q_heads) {
                        dst = reinterpret_cast<__half*>(r.q_out) + ((int64_t)m * r.num_q_heads + hd) * D;
                    } else {
                        const bool is_k = hd < r.num_q_heads + r.num_kv_heads;
                        const int kvh = hd - r.num_q_heads - (is_k ? 0 : r.num_kv_heads);
                        dst = reinterpret_cast<__half*>(is_k ? r.k_cache : r.v_cache) +
                              (int64_t)(base + r.kv_offset + m) * r.kv_tok_stride + (int64_t)kvh * r.kv_head_stride;
                    }
                    *reinterpret_cast<uint4*>(dst + d0) = *reinterpret_cast<const uint4*>(exch + row * kTileN + c0);
                }
            }
            named_bar_sync(bar, 128);
            return;
        }
        named_bar_sync(bar, 128);
        if (n_ok) {
            const int head = n / D, d = n - head * D;
            const bool rot = head < r.num_q_heads + r.num_kv_heads;
#pragma unroll
            for (int j = 0; j < 16; ++j) {
                if (j >= mcols) continue;
                const int m = m0 + j;
                __half o = h[j];
                if (rot) {
                    const int64_t pos = r.position_ids[(r.n_dev ? base + r.row_offset : 0) + m];
                    const __half c = reinterpret_cast<const __half*>(r.cos)[pos * D + d];
                    const __half sn = reinterpret_cast<const __half*>(r.sin)[pos * D + d];
                    const __half pr = exch[j * kTileN + (fl ^ half_d)];
                    // (x * cos) + (rotate_half(x) * sin): two products and one sum, each rounded (no fma)
                    o = __hadd_rn(__hmul_rn(h[j], c), __hmul_rn(d < half_d ? __hneg(pr) : pr, sn));
                }
                __half* dst;
                if (head < r.num_q_heads) {
                    dst = reinterpret_cast<__half*>(r.q_out) + ((int64_t)m * r.num_q_heads + head) * D;
                } else {
                    const bool is_k = head < r.num_q_heads + r.num_kv_heads;
                    const int kvh = head - r.num_q_heads - (is_k ? 0 : r.num_kv_heads);
                    dst = reinterpret_cast<__half*>(is_k ? r.k_cache : r.v_cache) +
                          (int64_t)(base + r.kv_offset + m) * r.kv_tok_stride + (int64_t)kvh * r.kv_head_stride;
                }
                dst[d] = o;
            }
        }
        named_bar_sync(bar, 128);
        return;
    }
    const bool n_ok = n < p.N_total;
    const int mcols = p.M - m0;                       // valid token columns of this chunk (may exceed 16)
    // fp16 outputs (plain store / residual add): the 16 x 128 tile goes through shared memory so that global memory
    // is touched with two independent 16-byte accesses per thread instead of one 2-byte access per token row.
    // Written as the plain per-row loop the residual loads compile into 13 serialised L2 round trips (4.2 us on the
    // tail of every o-proj / down-proj launch) and the stores into ~500 dependent instructions
    // (profiles/r1_gemm_tail_trace.txt).  y may alias the residual: all loads of the tile complete before any store.
    if ((p.mode == UMB_EPI_STORE || p.mode == UMB_EPI_RESIDUAL) && p.vec_ok) {
        const bool resid = p.mode == UMB_EPI_RESIDUAL;
        int row[2], col[2];
        bool ok[2];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int idx = fl + i * 128;
            row[i] = idx >> 4;
            col[i] = (idx & 15) * 8;
            ok[i] = row[i] < mcols && tile * kTileN + col[i] + 8 <= p.N_total;
        }
        if (resid) {
#pragma unroll
            for (int i = 0; i < 2; ++i)
                if (ok[i])
                    *reinterpret_cast<uint4*>(exch + row[i] * kTileN + col[i]) = *reinterpret_cast<const uint4*>(
                        p.residual + (int64_t)(m0 + row[i]) * p.ld_residual + tile * kTileN + col[i]);
            named_bar_sync(bar, 128);
        }
        const __half bb = (p.bias && n_ok) ? p.bias[n] : __float2half_rn(0.f);
        __half h[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) {
            h[j] = __float2half_rn(v[j]);
            if (p.bias) h[j] = __hadd(h[j], bb);
            if (resid) h[j] = __hadd(exch[j * kTileN + fl], h[j]);
        }
        if (resid) named_bar_sync(bar, 128);            // every thread has read its residual column
#pragma unroll
        for (int j = 0; j < 16; ++j) exch[j * kTileN + fl] = h[j];
        named_bar_sync(bar, 128);
#pragma unroll
        for (int i = 0; i < 2; ++i)
            if (ok[i])
                *reinterpret_cast<uint4*>(reinterpret_cast<__half*>(p.y) + (int64_t)(m0 + row[i]) * p.ldy + tile * kTileN + col[i]) =
                    *reinterpret_cast<const uint4*>(exch + row[i] * kTileN + col[i]);
        named_bar_sync(bar, 128);                       // the staging tile is free for the next chunk
        return;
    }
    if (!n_ok && !(p.mode == UMB_EPI_LOGITS && p.argmax)) return;
    const __half b = (p.bias && n_ok) ? p.bias[n] : __float2half_rn(0.f);
    // residual rows first, all loads in flight together: y may alias residual, so a load placed after a
    // store of the previous row would be serialised behind it (one L2 round trip per token row)
    __half res[16];
    if (p.mode == UMB_EPI_RESIDUAL) {
#pragma unroll
        for (int j = 0; j < 16; ++j)
            if (j < mcols) res[j] = p.residual[(int64_t)(m0 + j) * p.ld_residual + n];
    }
#pragma unroll
    for (int j = 0; j < 16; ++j) {
        if (j >= mcols) continue;
        const int m = m0 + j;
        __half h = __float2half_rn(v[j]);
        if (p.bias) h = __hadd(h, b);
        if (p.mode == UMB_EPI_RESIDUAL) {
            h = __hadd(res[j], h);
            reinterpret_cast<__half*>(p.y)[(int64_t)m * p.ldy + n] = h;
        } else if (p.mode == UMB_EPI_LOGITS) {
            const float f = __half2float(h);
            if (n_ok) reinterpret_cast<float*>(p.y)[(int64_t)m * p.ldy + n] = f;
            if (p.argmax) {
                // warp-level max first: one atomic per (warp, token)
                unsigned long long key =
                    n_ok ? (((unsigned long long)orderable_f32_g(f) << 32) | (unsigned int)(~n)) : 0ull;
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) {
                    const unsigned long long other = __shfl_xor_sync(0xffffffffu, key, o);
                    key = other > key ? other : key;
                }
                if ((threadIdx.x & 31) == 0) atomicMax(p.argmax + m, key);
            }
        } else {
            reinterpret_cast<__half*>(p.y)[(int64_t)m * p.ldy + n] = h;
        }
    }
}

// ------------------------------------------------------------------------------------------------
// host side: tensor maps
// ------------------------------------------------------------------------------------------------
typedef CUresult (*PFN_encodeTiled)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                    const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                    CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
static PFN_encodeTiled get_encode() {
    static PFN_encodeTiled fn = nullptr;
    static bool tried = false;
    if (!tried) {
        tried = true;
        void* sym = nullptr;
        cudaDriverEntryPointQueryResult qres;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &sym, cudaEnableDefault, &qres) == cudaSuccess &&
            qres == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<PFN_encodeTiled>(sym);
    }
    return fn;
}
// fp16 row-major x [rows, cols] as (64 cols, rows, cols / 64 atoms): box [64, box_rows, 2] = the two 128-byte-swizzled
// atoms of one 128-k slab in ONE copy
static int make_tmap_x3d(CUtensorMap* map, const void* base, uint64_t rows, uint64_t cols, uint64_t ld, uint32_t box_rows) {
    PFN_encodeTiled enc = get_encode();
    if (!enc) return UMB_ERR_DRIVER;
    const cuuint64_t dims[3] = {64, rows, cols / 64};
    const cuuint64_t strides[2] = {ld * sizeof(__half), 64 * sizeof(__half)};
    const cuuint32_t box[3] = {64, box_rows, 2};
    const cuuint32_t estr[3] = {1, 1, 1};
    const CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, const_cast<void*>(base), dims, strides, box, estr,
                           CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                           CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return arg_fail(__FILE__, __LINE__, "cuTensorMapEncodeTiled(3d)");
    return UMB_OK;
}

}  // namespace umb
