// (i) AWQ INT4 weight-dequant fused into a tcgen05 tensor-core GEMM, plus its fp16-weight twin.
//
// Replaces awq_ext.gemm_forward_cuda / dequantize_weights_cuda as called from AwqLinear.apply
// (reference umbrella/quantization/awq_utils.py:63-86) and torch F.linear for fp16 weights
// (lm_head: umbrella/models/llama.py:321; fp16 models: llama.py:87-110).
//
// Orientation ("swap-AB"): the verify pass multiplies M <= 128 token rows by a huge weight matrix,
// so the WEIGHTS are the UMMA A operand (128 output features per tile = the 128 TMEM lanes) and the
// token rows are the UMMA B/N operand (N = M padded to 16/32/64/128; AWQ beyond 128 rows: gemm_wide.cu):
//     D[128 features, MPAD tokens] (fp32, TMEM) += A[128, k] * B[MPAD, k]^T .
// Every weight byte is read from HBM exactly once per call.
//
// AWQ mainloop (per 128-feature x 128-k "unit" = one 8512-byte record of the repacked stream):
//   warp 0      TMA producer: cp.async.bulk of the packed record + cp.async.bulk.tensor (SW128)
//               of the x slab [MPAD, 128 k] into a kStages-deep shared-memory ring
//   warps 2..13 dequant, three groups of four warps taking units round-robin: thread = one feature
//               row x 128 k; one lop3 per nibble pair -> fp16 (1024+q | 1024+16q), an exact
//               hsub2 / hfma2 removes the bias and the zero point, one hmul2 by the group scale
//               == fp16((q - z) * s), the same rounding as the reference kernels; the fp16 row
//               goes straight to TENSOR MEMORY with tcgen05.st (no shared-memory round trip)
//   warp 1      one thread issues tcgen05.mma kind::f16 with A from TMEM, B from shared memory
//   warps 2..5  epilogue: tcgen05.ld the fp32 accumulator, fuse bias / residual / SiLU*up / fp32
//               logits, fp16 rounding placed where the reference has fp16 tensors
// Work is distributed stream-K: the (tile, k-group) space is cut into gridDim.x equal contiguous
// ranges (one persistent CTA per SM), partial tiles are reduced through a small fp32 workspace in a
// fixed order by the last-arriving CTA, so results are deterministic.
#include <cuda.h>
#include <stdio.h>
#include <stdlib.h>

#include "common.cuh"
#include "gemm_core.cuh"
#include "internal.h"

namespace umb {

#ifndef UMB_DQ_GROUPS
#define UMB_DQ_GROUPS 3
#endif
#ifndef UMB_DQ_GROUPS_16
#define UMB_DQ_GROUPS_16 UMB_DQ_GROUPS     // dequant groups of the <= 16-row instantiation (the verify pass of the static trees)
#endif
constexpr int kDqGroups = UMB_DQ_GROUPS;   // dequant warp groups (4 warps each, one per TMEM lane quarter)
constexpr int kGemmThreadsF16 = 96 + 128;           // producer + 2 MMA issuers + 4 epilogue warps (fp16 weights); AWQ: GemmCfg::kThreadsAwq
constexpr int kTmemCols = 512;
#ifndef UMB_WAIT_HINT
#define UMB_WAIT_HINT 1                    // 1: mbarrier waits carry a suspend-time hint (short in the pipeline, long in the epilogue)
#endif
#if UMB_WAIT_HINT
#define UMB_WAIT(bar, parity) mbar_wait_hint(bar, parity, 2000u)
#define UMB_WAIT_LONG(bar, parity) mbar_wait_hint(bar, parity, 100000u)
#else
#define UMB_WAIT(bar, parity) mbar_wait(bar, parity)
#define UMB_WAIT_LONG(bar, parity) mbar_wait(bar, parity)
#endif
// Pipeline variants that were built, measured on B200 and rejected (sleeping mbarrier polls in the idle warps,
// software-pipelined dequant, x slabs ahead of the weight ring, early residual fetch / early partial-sum
// reduction, a fourth dequant group) are recorded in profiles/r1_gemm_experiments.txt; none beat this form,
// whose steady state is bound by the fp16x2 issue rate of the dequant warps (scripts/ubench/pipe_rates.cu).

// ------------------------------------------------------------------------------------------------
// repack / dequantize / unpack
// ------------------------------------------------------------------------------------------------
__device__ __forceinline__ int64_t packed_row(int n, int row_block, int row_stride, int row_offset) {
    return (int64_t)(n / row_block) * row_stride + row_offset + n % row_block;
}

// thread (kw, c): 8 k x 8 n block of the checkpoint -> 8 words (one per n) of 8 k-nibbles
__global__ void awq_repack_weights_kernel(const int32_t* __restrict__ qweight, int K, int N, unsigned char* packed,
                                          int row_block, int row_stride, int row_offset) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    const int kw = blockIdx.y;
    if (c >= N / 8) return;
    uint32_t in[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) in[i] = (uint32_t)qweight[(int64_t)(kw * 8 + i) * (N / 8) + c];
    const int k0 = kw * 8, g = k0 / kGroup, kk = k0 % kGroup;
    const int kb = kk >> 6, ch = (kk >> 5) & 1, w = (kk >> 3) & 3;
    const int G = K / kGroup;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        uint32_t out = 0;
#pragma unroll
        for (int i = 0; i < 8; ++i) out |= ((in[i] >> (4 * nib_pos(j))) & 0xFu) << (4 * nib_pos(i));
        const int64_t pr = packed_row(c * 8 + j, row_block, row_stride, row_offset);
        const int64_t tile = pr / kTileN;
        const int r = (int)(pr % kTileN);
        unsigned char* rec = packed + (tile * G + g) * kRecordStride;
        *reinterpret_cast<uint32_t*>(rec + ((kb * 2 + ch) * kTileN + r) * 16 + w * 4) = out;
    }
}
// thread (g, c): scales and zeros of 8 consecutive output features of one group
__global__ void awq_repack_meta_kernel(const int32_t* __restrict__ qzeros, const __half* __restrict__ scales, int K,
                                       int N, unsigned char* packed, int row_block, int row_stride, int row_offset) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    const int g = blockIdx.y;
    if (c >= N / 8) return;
    const int G = K / kGroup;
    const uint32_t zin = (uint32_t)qzeros[(int64_t)g * (N / 8) + c];
    uint32_t zout = 0;
#pragma unroll
    for (int j = 0; j < 8; ++j) zout |= ((zin >> (4 * nib_pos(j))) & 0xFu) << (4 * j);
    const int64_t pr = packed_row(c * 8, row_block, row_stride, row_offset);   // 8-aligned run of rows
    const int64_t tile = pr / kTileN;
    const int r = (int)(pr % kTileN);
    unsigned char* rec = packed + (tile * G + g) * kRecordStride;
    *reinterpret_cast<uint32_t*>(rec + kRecZeroOff + (r >> 3) * 4) = zout;
    *reinterpret_cast<uint4*>(rec + kRecScaleOff + r * 2) =
        *reinterpret_cast<const uint4*>(scales + (int64_t)g * N + c * 8);
}

// awq_ext.dequantize_weights_cuda: out[k, n] = fp16((q - z) * s), checkpoint layout in, [K, N] out
__global__ void awq_dequantize_kernel(const int32_t* __restrict__ qweight, const int32_t* __restrict__ qzeros,
                                      const __half* __restrict__ scales, int K, int N, __half* __restrict__ out) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    const int k = blockIdx.y;
    if (c >= N / 8) return;
    const uint32_t q = (uint32_t)qweight[(int64_t)k * (N / 8) + c];
    const uint32_t z = (uint32_t)qzeros[(int64_t)(k / kGroup) * (N / 8) + c];
    union { uint4 u; __half h[8]; } s, o;
    s.u = *reinterpret_cast<const uint4*>(scales + (int64_t)(k / kGroup) * N + c * 8);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const int d = (int)((q >> (4 * nib_pos(j))) & 0xFu) - (int)((z >> (4 * nib_pos(j))) & 0xFu);
        o.h[j] = __hmul(__int2half_rn(d), s.h[j]);
    }
    *reinterpret_cast<uint4*>(out + (int64_t)k * N + c * 8) = o.u;
}

// packed stream -> fp16 [N_total, K]  (row = packed row); thread = (row, 8 k)
__global__ void awq_unpack_kernel(const unsigned char* __restrict__ packed, int K, int N_total,
                                  __half* __restrict__ out) {
    const int kw = blockIdx.x * blockDim.x + threadIdx.x;
    const int pr = blockIdx.y;
    if (kw >= K / 8) return;
    const int G = K / kGroup;
    const int k0 = kw * 8, g = k0 / kGroup, kk = k0 % kGroup;
    const int kb = kk >> 6, ch = (kk >> 5) & 1, w = (kk >> 3) & 3;
    const int tile = pr / kTileN, r = pr % kTileN;
    const unsigned char* rec = packed + ((int64_t)tile * G + g) * kRecordStride;
    const uint32_t word = *reinterpret_cast<const uint32_t*>(rec + ((kb * 2 + ch) * kTileN + r) * 16 + w * 4);
    const uint32_t zw = *reinterpret_cast<const uint32_t*>(rec + kRecZeroOff + (r >> 3) * 4);
    const int z = (int)((zw >> (4 * (r & 7))) & 0xFu);
    const __half s = *reinterpret_cast<const __half*>(rec + kRecScaleOff + r * 2);
    union { uint4 u; __half h[8]; } o;
#pragma unroll
    for (int i = 0; i < 8; ++i) o.h[i] = __hmul(__int2half_rn((int)((word >> (4 * nib_pos(i))) & 0xFu) - z), s);
    *reinterpret_cast<uint4*>(out + (int64_t)pr * K + k0) = o.u;
}

__device__ __forceinline__ unsigned long long gtimer() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t) : : "memory");
    return t;
}
// The timeline stamps are compiled in only for the `trace` variant build (-DUMB_GEMM_TRACE_BUILD=1,
// scripts/gemm_trace.py): even a predicated-off stamp costs issue slots inside the dequant loop.
#ifdef UMB_GEMM_TRACE_BUILD
#define UMB_TRACE(slot) do { if (p.trace) p.trace[(size_t)blockIdx.x * 16 + (slot)] = gtimer(); } while (0)
#else
#define UMB_TRACE(slot) do { } while (0)
#endif

template <int MPAD>
struct GemmCfg {
    // 128 rows (AWQ): weight records and x slabs in rings of their own.  A shared ring holds four units of 41 KB, and a unit
    // occupies its place from the request over the dequantisation to the product.  The records' ring is free as soon as they
    // are in registers, so dequantisation runs ahead of the slabs: 500 rows in four passes through a layer of width 4096 and its head
    // 887 -> 849 us; with the heads of split tiles reduced by every group of warps (below) 683.
    static constexpr bool kSplit = MPAD >= 128;
    // dequant groups per CTA (AWQ).  kSplit takes two: every ring depth is a multiple of it, so a stage always comes back to
    // the group that used it last, which the parity waits need there (see the dequant warps' note)
    static constexpr int kDq = MPAD == 16 ? UMB_DQ_GROUPS_16 : (kSplit ? 2 : kDqGroups);
    static constexpr int kWStages = 6;                                              // records held with kSplit
    static constexpr int kThreadsAwq = 96 + 128 * (kDq + 1) + (kSplit ? 32 : 0);   // (the x slabs' own warp)
    static constexpr int kStagesAwq = MPAD == 16 ? 10 : (MPAD == 32 ? 8 : (MPAD == 64 ? 6 : 4));
    static constexpr int kStagesF16 = MPAD <= 32 ? 8 : (MPAD == 64 ? 6 : 4);
    static constexpr int kXBytesAwq = MPAD * 256;           // [2 atoms][MPAD][128 B]
    static constexpr int kXBytesF16 = MPAD * 128;           // [MPAD][128 B]
    static constexpr int kWBytesF16 = kTileN * 128;         // [128][128 B]
    static constexpr int kPackedStride = 8576;              // record padded to a 128-byte multiple
    // epilogue staging: output tile + cos / sin rows (RoPE), for each group of warps that finishes tiles
    static constexpr int kExchBytes = 3 * 16 * 128 * 2;
    // (AWQ) all of them reduce the head of a split tile.  From four chunks of 16 columns on (a layer of width 4096 and its head:
    // 40 rows 254 -> 237 us, 64 rows 262 -> 239); up to 32 rows are one or two chunks, hardly more than one group's turn.
    static constexpr bool kShare = MPAD >= 64;
    static constexpr int kExchGroups = kShare ? kDq + 1 : 1;
    // Independent fp32 accumulators in TMEM (columns a * MPAD): consecutive k-steps rotate through them so
    // that back-to-back tcgen05.mma never wait on each other's accumulate (a dependent 128xNx16 MMA chain
    // runs at its ~150-cycle latency, not at its 8-cycle issue rate); the epilogue sums them.
    static constexpr int kNumAcc = MPAD <= 16 ? 8 : (MPAD == 32 ? 4 : 2);
    static constexpr int kTmemACol0 = kNumAcc * MPAD < 128 ? 128 : kNumAcc * MPAD;   // A operand stages start here
    static constexpr int kTmemAStages = (kTmemCols - kTmemACol0) / 64;             // 6 (4 at MPAD = 128)
    static constexpr int kBarBytes = 576;
    static constexpr int smem_bytes(bool awq, int stages) {
        return 1024 /*align slack*/ + kBarBytes + kExchGroups * kExchBytes +
               (awq && kSplit ? stages * kXBytesAwq + kWStages * kPackedStride
                              : stages * (awq ? (kXBytesAwq + kPackedStride) : (kXBytesF16 + kWBytesF16)));
    }
};

// v[j] = sum over the accumulators of column (m0 + j), in a fixed order (deterministic).  The
// accumulators are split between the two MMA warps (first / second half); `use_mask` bit w tells
// whether warp w issued anything into its half during this segment.
template <int kAcc, int MPAD>
__device__ __forceinline__ void load_acc_sum(uint32_t taddr, float (&v)[16], int use_mask) {
    uint32_t rr[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) v[j] = 0.f;
#pragma unroll
    for (int a = 0; a < kAcc; ++a) {
        if (!((use_mask >> (a / (kAcc / 2))) & 1)) continue;
        UMB_TMEM_LD_X16(taddr + a * MPAD, rr);
        tc_wait_ld();
#pragma unroll
        for (int j = 0; j < 16; ++j) v[j] += __uint_as_float(rr[j]);
    }
}

// Warp roles (AWQ: 19 warps, fp16: 7 warps)
//   warp 0        TMA producer.  The weight copies of the first kStages units are issued BEFORE
//                 griddepcontrol.wait (weights never depend on the stream predecessor), the x slabs after it
//   warps 1, 2    MMA issuers: CTA-local unit u is issued by warp 1 + (u & 1), each into its own half of
//                 the TMEM accumulators
//   warps 3..14   dequant groups (AWQ only): shared memory -> registers -> tensor memory; they start as
//                 soon as a weight record has landed, also before the predecessor kernel has finished
//   last 4 warps  epilogue only (AWQ: warps 15..18, fp16: warps 3..6): the partial-tile fix-up is a chain of
//                 global round trips and must not stall the dequant stream
//   65..128 rows  (AWQ) two dequant groups, warps 3..10, which also reduce when they have no units left; epilogue warps
//                 11..14; warp 15 requests the x slabs
template <int MPAD, bool kAwq>
__global__ void __launch_bounds__(kAwq ? GemmCfg<MPAD>::kThreadsAwq : kGemmThreadsF16, 1)
gemm_kernel(const __grid_constant__ CUtensorMap tmap_x, const __grid_constant__ CUtensorMap tmap_w,
            const GemmParams p) {
    using Cfg = GemmCfg<MPAD>;
    const int kStages = p.stages;
    constexpr int kXBytes = kAwq ? Cfg::kXBytesAwq : Cfg::kXBytesF16;
    constexpr int kWStride = kAwq ? Cfg::kPackedStride : Cfg::kWBytesF16;
    constexpr uint32_t kWTxBytes = kAwq ? (uint32_t)kRecordBytes : (uint32_t)Cfg::kWBytesF16;
    constexpr uint32_t kIdesc = umma_idesc_f16(kTileN, MPAD);
    constexpr int kNumAcc = Cfg::kNumAcc;                       // >= 2, even
    constexpr int kAccUsed = kAwq ? kNumAcc : (kNumAcc < 8 ? kNumAcc : 8);
    constexpr int kAccHalf = kAccUsed / 2;                      // accumulators per MMA warp
    constexpr int kACol0 = Cfg::kTmemACol0;
    constexpr int kAStages = Cfg::kTmemAStages;
    // the MMA warps take alternate units, so a ring stage must always come back to the same warp (parity waits, see the
    // dequant warps' note): both rings need an even depth
    static_assert(!kAwq || (kAStages % 2 == 0 && Cfg::kStagesAwq % 2 == 0), "ring depths must be even");
    constexpr bool kSplit = kAwq && Cfg::kSplit, kShare = kAwq && Cfg::kShare;
    static_assert(!kSplit || (kAStages % Cfg::kDq == 0 && Cfg::kWStages % Cfg::kDq == 0 && Cfg::kStagesAwq == kAStages),
                  "the rings of separate records must return each stage to its dequant group");
    const int kWRing = kSplit ? Cfg::kWStages : kStages;        // depth of the weight records' ring
    constexpr int kDq = Cfg::kDq;                               // dequant groups of this CTA
    constexpr int kFinish = kShare ? Cfg::kExchGroups : 1;      // groups of warps that reduce the head of a split tile

    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    unsigned char* s_x = smem;                                   // kStages x kXBytes   (1024-aligned slabs)
    unsigned char* s_w = s_x + kStages * kXBytes;                // kStages x kWStride
    __half* s_exch = reinterpret_cast<__half*>(s_w + kWRing * kWStride);
    uint64_t* bars = reinterpret_cast<uint64_t*>(reinterpret_cast<unsigned char*>(s_exch) + Cfg::kExchGroups * Cfg::kExchBytes);
    uint64_t* full_w = bars;                  // [kStages]   weight record / tile landed
    uint64_t* full_x = bars + 16;             // [kStages]   x slab landed
    uint64_t* done = bars + 32;               // [kStages]   every MMA of the unit in this stage has retired
    uint64_t* a_full = bars + 48;             // [kAStages]  dequantised A operand is in tensor memory
    uint64_t* acc_full = bars + 56;
    uint64_t* acc_empty = bars + 57;
    uint32_t* s_tmem = reinterpret_cast<uint32_t*>(bars + 58);
    uint64_t* last_full = bars + 59;          //             kShare: the last segment's accumulators are complete
    uint64_t* w_empty = bars + 60;            // [kWStages]  kSplit: the record in this stage is in the dequant group's registers

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) UMB_TRACE(0);
    const long long U = (long long)p.tiles * p.units_per_tile, P = gridDim.x;
    const long long u_begin = sk_begin(blockIdx.x, U, P), u_end = sk_begin(blockIdx.x + 1, U, P);
    const int n_units = (int)(u_end - u_begin);
    const int in_tile0 = (int)u_begin % p.units_per_tile;        // position of the first unit inside its tile
    const int tile0 = (int)u_begin / p.units_per_tile;

    if (warp == 0 && lane == 0) {
        tma_prefetch_desc(&tmap_x);
        tma_prefetch_desc(&tmap_w);
        for (int i = 0; i < kStages; ++i) {
            if (!kSplit) mbar_init(full_w + i, 1);
            mbar_init(full_x + i, 1);
            mbar_init(done + i, 1);
        }
        for (int i = 0; kSplit && i < kWRing; ++i) {
            mbar_init(full_w + i, 1);
            mbar_init(w_empty + i, 4);
        }
        for (int i = 0; i < kAStages; ++i) mbar_init(a_full + i, 4);
        mbar_init(acc_full, 2);
        if (kShare) mbar_init(last_full, 2);
        mbar_init(acc_empty, 4);
        fence_barrier_init();
    }
    if (warp == 1) {
        tmem_alloc(s_tmem, kTmemCols);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    pdl_launch_dependents();
    const uint32_t tmem_base = *s_tmem;
    if (threadIdx.x == 0) UMB_TRACE(1);

    if (warp == 0) {
        // ===================== TMA producer (whole warp runs the loop, one elected lane issues) =====================
        const uint64_t pol_w = l2_policy_evict_first(), pol_x = l2_policy_evict_last();
        const unsigned char* src = p.packed + (kAwq ? u_begin * kRecordStride : 0);
        const int n_pre = n_units < kWRing ? n_units : kWRing;
        // The weight copies of the whole ring are requested before griddepcontrol.wait (they never depend on the
        // stream predecessor), the x slabs after it.  (Requesting only a few records early, so that the first x
        // slab does not queue behind ~85 KB of weights, starts the first MMA 2 us sooner but measured no faster:
        // the dequant warps set the pace.)
        const int n_early = n_pre;
        int tile = tile0, g = in_tile0;                          // (tile, g) of the next weight copy
        auto issue_w = [&](int stage) {
            mbar_arrive_expect_tx(full_w + stage, kWTxBytes);
            if constexpr (kAwq)
                tma_bulk_g2s(s_w + stage * kWStride, src, kRecordBytes, full_w + stage, pol_w);
            else
                tma_tensor2d_g2s(s_w + stage * kWStride, &tmap_w, g * 64, tile * kTileN, full_w + stage, pol_w);
        };
        auto issue_x = [&](int stage, int gk) {
            if (kSplit) return;                                   // requested by the x slabs' own warp
            mbar_arrive_expect_tx(full_x + stage, (uint32_t)kXBytes);
            unsigned char* xs = s_x + stage * kXBytes;
            if constexpr (kAwq) {
                tma_tensor3d_g2s(xs, &tmap_w, 0, 0, gk * 2, full_x + stage, pol_x);      // tmap_w = x as [64, rows, K / 64]
            } else {
                tma_tensor2d_g2s(xs, &tmap_x, gk * 64, 0, full_x + stage, pol_x);
            }
        };
        auto advance_w = [&]() {
            src += kRecordStride;
            if (++g == p.units_per_tile) {
                g = 0;
                ++tile;
            }
        };
        for (int i = 0; i < n_early; ++i) {                      // weights first: independent of the predecessor
            if (elect_one()) issue_w(i);
            __syncwarp();
            advance_w();
        }
        if (lane == 0) UMB_TRACE(2);
        pdl_wait();                                              // x is the predecessor's output
        if (lane == 0) UMB_TRACE(3);
        int gx = in_tile0;
        for (int i = 0; i < n_early; ++i) {
            if (elect_one()) issue_x(i, gx);
            __syncwarp();
            if (++gx == p.units_per_tile) gx = 0;
        }
        for (int i = n_early; i < n_pre; ++i) {                  // rest of the ring: stages still untouched
            if (elect_one()) {
                issue_w(i);
                issue_x(i, g);
            }
            __syncwarp();
            advance_w();
        }
        Ring r;
        r.phase = 1;                                             // every stage has been used once
        for (int i = n_pre; i < n_units; ++i) {
            // the unit that last used this stage has retired (kSplit: its record has been read)
            if constexpr (kSplit) UMB_WAIT(w_empty + r.stage, r.phase ^ 1);
            else UMB_WAIT(done + r.stage, r.phase ^ 1);
            if (elect_one()) {
                issue_w(r.stage);
                issue_x(r.stage, g);
            }
            __syncwarp();
            advance_w();
            r.advance(kWRing);
        }
        if (lane == 0) UMB_TRACE(10);
    } else if (kSplit && warp == GemmCfg<MPAD>::kThreadsAwq / 32 - 1) {
        // ===================== x-slab producer (AWQ, kSplit) =====================
        const uint64_t pol_x = l2_policy_evict_last();
        pdl_wait();                                              // x is the predecessor's output
        int gx = in_tile0, stage = 0, use = 0;
        for (int i = 0; i < n_units; ++i) {
            if (use > 0) UMB_WAIT(done + stage, (use - 1) & 1); // the unit that last used this stage has retired
            if (elect_one()) {
                mbar_arrive_expect_tx(full_x + stage, (uint32_t)kXBytes);
                tma_tensor3d_g2s(s_x + stage * kXBytes, &tmap_w, 0, 0, gx * 2, full_x + stage, pol_x);
            }
            __syncwarp();
            if (++gx == p.units_per_tile) gx = 0;
            if (++stage == kStages) {
                stage = 0;
                ++use;
            }
        }
    } else if (warp <= 2) {
        // ===================== MMA issuers: warp 1 takes even CTA-local units, warp 2 odd ones =====================
        const int par = warp - 1;
        const uint32_t d_base = tmem_base + par * kAccHalf * MPAD;   // this warp's accumulators
        constexpr uint64_t kDescHi = ((uint64_t)(1024 >> 4) << 32) | ((uint64_t)1 << 46) | ((uint64_t)2 << 61) | ((uint64_t)1 << 16);
        int st = par % kStages, ph = (par / kStages) & 1;            // smem ring position of unit `u`
        int ts = par % kAStages, pa = 0;                              // tensor-memory A ring position
        int u = par, seg = 0, seg_begin = 0, in_tile = in_tile0;
        while (seg_begin < n_units) {
            const int seg_end = seg_begin + min(n_units - seg_begin, p.units_per_tile - in_tile);
            UMB_WAIT_LONG(acc_empty, (seg & 1) ^ 1);
            tc_fence_after();
            bool first = true;
            for (; u < seg_end; u += 2) {
                const bool last = u + 2 >= seg_end;
                if constexpr (kAwq) {
                    UMB_WAIT(a_full + ts, pa);
                } else {
                    UMB_WAIT(full_w + st, ph);
                }
                UMB_WAIT(full_x + st, ph);
                tc_fence_after();
                if (u == 0 && lane == 0) UMB_TRACE(5);
                const uint32_t xs = smem_u32(s_x + st * kXBytes);
                const uint64_t bd0 = kDescHi | (uint64_t)((xs & 0x3FFFF) >> 4);
                if constexpr (kAwq) {
                    const uint32_t a_col = tmem_base + kACol0 + ts * 64;
                    if (elect_one()) {
#pragma unroll
                        for (int kk = 0; kk < 8; ++kk) {
                            const uint64_t bd = bd0 + (uint64_t)(((kk >> 2) * (MPAD * 128) + (kk & 3) * 32) >> 4);
                            umma_ts_f16(d_base + (kk % kAccHalf) * MPAD, a_col + kk * 8, bd, kIdesc,
                                        (first && kk < kAccHalf) ? 0u : 1u);
                        }
                        umma_commit(done + st);
                        if (last) umma_commit(acc_full);
                        if (kShare && last && seg_end == n_units) umma_commit(last_full);
                    }
                } else {
                    const uint32_t ws = smem_u32(s_w + st * kWStride);
                    const uint64_t ad0 = kDescHi | (uint64_t)((ws & 0x3FFFF) >> 4);
                    if (elect_one()) {
#pragma unroll
                        for (int kk = 0; kk < 4; ++kk)
                            umma_ss_f16(d_base + (kk % kAccHalf) * MPAD, ad0 + kk * 2, bd0 + kk * 2, kIdesc,
                                        (first && kk < kAccHalf) ? 0u : 1u);
                        umma_commit(done + st);
                        if (last) umma_commit(acc_full);
                    }
                }
                __syncwarp();
                first = false;
                st += 2;
                while (st >= kStages) {
                    st -= kStages;
                    ph ^= 1;
                }
                ts += 2;
                if (ts >= kAStages) {
                    ts -= kAStages;
                    pa ^= 1;
                }
            }
            if (first) {                     // this warp had no unit in the segment: plain arrival
                if (elect_one()) {
                    mbar_arrive(acc_full);
                    if (kShare && seg_end == n_units) mbar_arrive(last_full);
                }
                __syncwarp();
            }
            seg_begin = seg_end;
            in_tile = 0;
            ++seg;
        }
        if (par == 0 && lane == 0) UMB_TRACE(6);
    } else {
        const int q = warp & 3;                      // TMEM lane quarter this warp may touch
        const int grp = (warp - 3) >> 2;             // AWQ: dequant group 0..kDqGroups-1, then the epilogue group
        const bool is_epi = kAwq ? (grp == kDq) : true;
        const int fl = q * 32 + lane;                // feature lane 0..127
        const uint32_t lane_addr = (uint32_t)(q * 32) << 16;
        // acc[j] += the partial sums the other CTAs of `tile_` published for token columns [m0, m0 + 16), in
        // ascending CTA order (deterministic); the polled words are stored back as zeros.
        auto reduce_others = [&](float (&acc)[16], int m0, int tile_, int c_first, int n_other) {
            const int mcols = p.M - m0;
            uint32_t* sl0 = reinterpret_cast<uint32_t*>(p.slots) +
                            ((size_t)tile_ + c_first + 1) * (MPAD * kTileN) + m0 * kTileN + fl;
            if (mcols <= 4) {
                // few token rows (draft levels): 8 slots in flight per round trip
                for (int c0 = 0; c0 < n_other; c0 += 8) {
                    uint32_t t[8][4];
                    bool pending;
                    do {
                        pending = false;
#pragma unroll
                        for (int cc = 0; cc < 8; ++cc)
#pragma unroll
                            for (int j = 0; j < 4; ++j) {
                                const bool need = c0 + cc < n_other && j < mcols;
                                t[cc][j] = need ? ld_relaxed_gpu_u32(sl0 + (size_t)(c0 + cc) * (MPAD * kTileN) + j * kTileN) : 0x80000000u;
                            }
#pragma unroll
                        for (int cc = 0; cc < 8; ++cc)
#pragma unroll
                            for (int j = 0; j < 4; ++j) pending |= t[cc][j] == 0u;
                    } while (pending);
#pragma unroll
                    for (int cc = 0; cc < 8; ++cc)
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            acc[j] += __uint_as_float(t[cc][j]);
                            if (c0 + cc < n_other && j < mcols) sl0[(size_t)(c0 + cc) * (MPAD * kTileN) + j * kTileN] = 0u;
                        }
                }
            } else if (mcols > 0) {
                for (int c0 = 0; c0 < n_other; c0 += 2) {
                    uint32_t t[2][16];
                    bool pending;
                    do {
                        pending = false;
#pragma unroll
                        for (int cc = 0; cc < 2; ++cc)
#pragma unroll
                            for (int j = 0; j < 16; ++j) {
                                const bool need = c0 + cc < n_other && j < mcols;
                                t[cc][j] = need ? ld_relaxed_gpu_u32(sl0 + (size_t)(c0 + cc) * (MPAD * kTileN) + j * kTileN) : 0x80000000u;
                            }
#pragma unroll
                        for (int cc = 0; cc < 2; ++cc)
#pragma unroll
                            for (int j = 0; j < 16; ++j) pending |= t[cc][j] == 0u;
                    } while (pending);
#pragma unroll
                    for (int cc = 0; cc < 2; ++cc)
#pragma unroll
                        for (int j = 0; j < 16; ++j) {
                            acc[j] += __uint_as_float(t[cc][j]);
                            if (c0 + cc < n_other && j < mcols) sl0[(size_t)(c0 + cc) * (MPAD * kTileN) + j * kTileN] = 0u;
                        }
                }
            }
        };
        // The reducer's share of a tile: chunks of 16 token columns m_first, m_first + m_step, ...
        auto reduce_tile = [&](int m_first, int m_step, int tile_, int c_first, int c_last, int use_mask, __half* ex, uint32_t bar) {
#pragma unroll 1
            for (int m0 = m_first; m0 < MPAD; m0 += m_step) {
                if (!(m0 < p.M || p.mode == UMB_EPI_SILU_MUL || p.mode == UMB_EPI_ROPE_QKV)) break;
                float v[16];
                load_acc_sum<kAccUsed, MPAD>(tmem_base + lane_addr + m0, v, use_mask);
                reduce_others(v, m0, tile_, c_first, c_last - c_first);
                epilogue_chunk(p, tile_, fl, m0, v, ex, bar);
            }
        };
        if (!is_epi) {
            // ===================== dequant warps (AWQ): group g takes CTA-local units g, g + kDqGroups, ... =====================
            if constexpr (kAwq) {
                int dq_st = grp % kWRing, dq_ph = 0, dq_ts = grp % kAStages;      // ring positions of unit `mine`
                int w_first = grp;                                                 // first unit of this group that re-uses a TMEM stage
                while (w_first < kAStages) w_first += kDq;
                int w_st = (w_first - kAStages) % kStages, w_ph = 0;               // ring position of unit `mine - kAStages`
                // the packed words / scale / zero of a unit are pulled into registers as soon as its record has landed
                uint4 w4[4];
                uint32_t sbits = 0, zw = 0;
                auto fetch = [&](int st_) {
                    const uint32_t rec = smem_u32(s_w + st_ * kWStride);
#pragma unroll
                    for (int c = 0; c < 4; ++c) w4[c] = lds128(rec + (c * kTileN + fl) * 16);    // 128 k of this feature row
                    sbits = lds16(rec + kRecScaleOff + fl * 2);
                    zw = lds32(rec + kRecZeroOff + (fl >> 3) * 4);
                };
                if (grp < n_units) {
                    UMB_WAIT(full_w + dq_st, dq_ph);
                    if (grp == 0 && q == 0 && lane == 0) UMB_TRACE(4);
                    fetch(dq_st);
                    if constexpr (kSplit) {
                        __syncwarp();
                        if (lane == 0) mbar_arrive(w_empty + dq_st);
                    }
                }
                for (int mine = grp; mine < n_units; mine += kDq) {
                    const int ts = dq_ts;
                    dq_st += kDq;
                    if (dq_st >= kWRing) {
                        dq_st -= kWRing;
                        dq_ph ^= 1;
                    }
                    dq_ts += kDq;
                    if (dq_ts >= kAStages) dq_ts -= kAStages;
                    const uint32_t z = (zw >> (4 * (fl & 7))) & 0xFu;
                    const __half2 ce = as_h2((0x6400u | z) * 0x10001u);                 // (1024 + z) x2
                    const __half2 neg_co = as_h2((0xD400u | (z << 4)) * 0x10001u);      // -(64 + z) x2
                    const __half2 s2 = as_h2(sbits * 0x10001u);
                    const uint32_t magic = 0x64006400u;
                    const uint32_t taddr = tmem_base + lane_addr + kACol0 + ts * 64;
#pragma unroll
                    for (int c = 0; c < 4; ++c) {                            // 4 chunks of 32 k (16 TMEM columns)
                        const uint32_t words[4] = {w4[c].x, w4[c].y, w4[c].z, w4[c].w};
                        uint32_t a[16];
#pragma unroll
                        for (int w = 0; w < 4; ++w) dequant_word(words[w], magic, ce, neg_co, s2, &a[w * 4]);
                        UMB_TMEM_ST_X16(taddr + c * 16, a);
                    }
                    tc_wait_st();
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(a_full + ts);
                    if (mine + kDq < n_units) {            // this group's next unit v: (dq_st, dq_ph) already point at it
                        // (1) The unit that last used v's tensor-memory stage (v - kAStages) must have retired before the
                        //     stage is overwritten.
                        // (2) The same wait makes the parity wait on full_w sound.  A parity wait lets a waiter through that
                        //     is TWO uses ahead of its barrier (the parity of "use j - 2 completed" equals that of "use j
                        //     completed"), and the previous occupant of v's shared-memory stage, unit v - kStages, belongs to
                        //     another group: with the 4-deep ring of the 128-column instantiation it is unit mine - 1, which
                        //     may still be in flight.  The group then read a stale record and signalled a_full early, the MMA
                        //     retired early, and the producer re-armed full_w while its previous copy was still open: the
                        //     "Warp Illegal Instruction" that killed one 128-row launch in ~150 (profiles/r2_m128_root_cause.txt).
                        //     done[v - kAStages] implies done[v - kStages]: both ring depths are even, so the two units were
                        //     issued and committed, in order, by the same MMA thread; a retired occupant has landed, so
                        //     full_w is at most one use behind.  (v < kAStages: first use of both stages, nothing to wait for.)
                        //     kSplit: the producer no longer orders the records behind done, so (1) itself has to know that
                        //     done[v - 2 kAStages] is over, and (2) that record v - kWStages was read: this group has waited
                        //     for both itself, both depths being multiples of the number of groups.
                        if (mine + kDq >= kAStages) {
                            UMB_WAIT(done + w_st, w_ph);
                            tc_fence_after();
                            w_st += kDq;
                            if (w_st >= kStages) {
                                w_st -= kStages;
                                w_ph ^= 1;
                            }
                        }
                        UMB_WAIT(full_w + dq_st, dq_ph);
                        fetch(dq_st);
                        if constexpr (kSplit) {
                            __syncwarp();
                            if (lane == 0) mbar_arrive(w_empty + dq_st);
                        }
                    }
                }
                if constexpr (kShare) {
                    // The head of a split tile is reduced by all groups of warps, one chunk of 16 columns each in turn: a chunk
                    // waits for two or three round trips to the other CTAs' sums, 24 of them in series with one group
                    // when five CTAs share a tile (849 -> 683 us, see kSplit; four sums in flight a thread instead of two
                    // spill registers: 753).
                    const int tile_ = (int)((u_end - 1) / p.units_per_tile);
                    const long long tile_u0 = (long long)tile_ * p.units_per_tile;
                    const int c_first = sk_owner(tile_u0, U, P), c_last = sk_owner(tile_u0 + p.units_per_tile - 1, U, P);
                    if (n_units > 0 && c_first == (int)blockIdx.x && c_last != c_first) {
                        const int begin = tile_u0 > u_begin ? (int)(tile_u0 - u_begin) : 0;       // CTA-local first unit of the segment
                        const int n_odd = (n_units >> 1) - (begin >> 1);
                        const int use_mask = ((n_units - begin - n_odd) > 0 ? 1 : 0) | (n_odd > 0 ? 2 : 0);
                        pdl_wait();
                        UMB_WAIT_LONG(last_full, 0);
                        tc_fence_after();
                        reduce_tile(16 * (grp + 1), 16 * kFinish, tile_, c_first, c_last, use_mask,
                                    s_exch + (grp + 1) * (Cfg::kExchBytes / 2), 3 + grp);
                    }
                }
            }
        } else {
            // ===================== epilogue warps =====================
            const int ew = kAwq ? warp - 3 - 4 * kDq : warp - 3;       // 0..3 inside the epilogue group
            pdl_wait();                                  // residual / workspace / y belong to the predecessors
            if (ew == 0 && lane == 0) UMB_TRACE(11);
            int seg = 0, seg_begin = 0, in_tile = in_tile0, tile = tile0;
            while (seg_begin < n_units) {
                const int seg_end = seg_begin + min(n_units - seg_begin, p.units_per_tile - in_tile);
                const int seg_len = seg_end - seg_begin;
                const bool whole = seg_len == p.units_per_tile;
                // which MMA warps issued into their accumulators during this segment
                const int n_odd = (seg_end >> 1) - (seg_begin >> 1);               // odd CTA-local indices in [begin, end)
                const int use_mask = ((seg_len - n_odd) > 0 ? 1 : 0) | (n_odd > 0 ? 2 : 0);
                const long long tile_u0 = (long long)tile * p.units_per_tile;
                const int c_first = whole ? (int)blockIdx.x : sk_owner(tile_u0, U, P);
                const int c_last = whole ? (int)blockIdx.x : sk_owner(tile_u0 + p.units_per_tile - 1, U, P);
                const bool reducer = !whole && (int)blockIdx.x == c_first;
                UMB_WAIT_LONG(acc_full, seg & 1);
                tc_fence_after();
                if (ew == 0 && lane == 0) UMB_TRACE(seg == 0 ? 7 : 12);
                if (whole) {
#pragma unroll 1
                    for (int m0 = 0; m0 < MPAD; m0 += 16) {
                        float v[16];
                        load_acc_sum<kAccUsed, MPAD>(tmem_base + lane_addr + m0, v, use_mask);
                        if (m0 + 16 >= MPAD) {       // accumulators fully read: hand TMEM back to the MMA warps
                            tc_fence_before();
                            __syncwarp();
                            if (lane == 0) mbar_arrive(acc_empty);
                        }
                        if (m0 < p.M || p.mode == UMB_EPI_SILU_MUL || p.mode == UMB_EPI_ROPE_QKV)
                            epilogue_chunk(p, tile, fl, m0, v, s_exch);
                    }
                } else {
                    // Partial tile.  The CTA that owns the HEAD of the tile (c_first; that part is the last
                    // segment of its range) is the reducer; every other part is the FIRST segment of its owner,
                    // i.e. published early in the kernel.  Publication needs no fence, counter or barrier: every
                    // 32-bit word of a slot is its own flag (0 = not yet written; a partial sum of +0.0f is stored
                    // as -0.0f, which adds identically), the reducer polls exactly the words it needs with relaxed
                    // gpu-scope loads, adds them (ascending CTA order -- deterministic) and stores the zeros back,
                    // which leaves the workspace clean for the next launch.
                    if (!reducer) {
                        uint32_t* slot = reinterpret_cast<uint32_t*>(p.slots) + ((size_t)tile + blockIdx.x) * (MPAD * kTileN);
#pragma unroll 1
                        for (int m0 = 0; m0 < MPAD; m0 += 16) {
                            float v[16];
                            load_acc_sum<kAccUsed, MPAD>(tmem_base + lane_addr + m0, v, use_mask);
                            if (m0 + 16 >= MPAD) {
                                tc_fence_before();
                                __syncwarp();
                                if (lane == 0) mbar_arrive(acc_empty);
                            }
#pragma unroll
                            for (int j = 0; j < 16; ++j)
                                if (m0 + j < p.M) {
                                    const uint32_t u = __float_as_uint(v[j]);
                                    slot[(m0 + j) * kTileN + fl] = u ? u : 0x80000000u;
                                }
                        }
                    } else {
                        // always the CTA's last segment: the accumulators are not handed back
                        if (ew == 0 && lane == 0) UMB_TRACE(14);
                        reduce_tile(0, 16 * kFinish, tile, c_first, c_last, use_mask, s_exch, 2);
                        if (ew == 0 && lane == 0) UMB_TRACE(15);
                    }
                }
                seg_begin = seg_end;
                in_tile = 0;
                ++tile;
                ++seg;
                if (ew == 0 && lane == 0) UMB_TRACE(seg == 1 ? 8 : 13);
            }
        }
    }

    tc_fence_before();
    __syncthreads();
    if (threadIdx.x == 0) UMB_TRACE(9);
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem_base, kTmemCols);
    }
}

// ------------------------------------------------------------------------------------------------
// probe: one 128 x 16 x 64 UMMA, A from shared memory (mode 0) or tensor memory (mode 1)
// ------------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(128, 1)
probe_umma_kernel(const __half* __restrict__ a, const __half* __restrict__ b, float* __restrict__ d, int mode) {
    __shared__ __align__(1024) unsigned char s_a[128 * 128];
    __shared__ __align__(1024) unsigned char s_b[16 * 128];
    __shared__ uint64_t bar;
    __shared__ uint32_t s_tmem;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, r = threadIdx.x;
    // manual SW128 K-major tiles: element (row, k) at (row/8)*1024 + (row%8)*128 + ((k/8) ^ (row%8))*16 + (k%8)*2
    for (int c = 0; c < 8; ++c) {
        const uint4 va = *reinterpret_cast<const uint4*>(a + r * 64 + c * 8);
        *reinterpret_cast<uint4*>(s_a + (r >> 3) * 1024 + (r & 7) * 128 + ((c ^ (r & 7)) << 4)) = va;
        if (r < 16) {
            const uint4 vb = *reinterpret_cast<const uint4*>(b + r * 64 + c * 8);
            *reinterpret_cast<uint4*>(s_b + (r >> 3) * 1024 + (r & 7) * 128 + ((c ^ (r & 7)) << 4)) = vb;
        }
    }
    fence_proxy_async_smem();
    if (threadIdx.x == 0) {
        mbar_init(&bar, 1);
        fence_barrier_init();
    }
    if (warp == 0) {
        tmem_alloc(&s_tmem, 64);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = s_tmem;
    const uint32_t lane_addr = (uint32_t)(warp * 32) << 16;
    if (mode == 1) {
        uint32_t regs[32];
        for (int c = 0; c < 32; ++c) regs[c] = *reinterpret_cast<const uint32_t*>(a + r * 64 + c * 2);
        UMB_TMEM_ST_X16(tmem + lane_addr + 32, (&regs[0]));
        UMB_TMEM_ST_X16(tmem + lane_addr + 48, (&regs[16]));
        tc_wait_st();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (threadIdx.x == 0) {
        constexpr uint32_t idesc = umma_idesc_f16(128, 16);
        for (int kk = 0; kk < 4; ++kk) {
            const uint64_t bd = umma_smem_desc_sw128(smem_u32(s_b) + kk * 32);
            if (mode == 1) {
                umma_ts_f16(tmem, tmem + 32 + kk * 8, bd, idesc, kk ? 1u : 0u);
            } else {
                const uint64_t ad = umma_smem_desc_sw128(smem_u32(s_a) + kk * 32);
                umma_ss_f16(tmem, ad, bd, idesc, kk ? 1u : 0u);
            }
        }
        umma_commit(&bar);
    }
    mbar_wait(&bar, 0);
    tc_fence_after();
    uint32_t rr[16];
    UMB_TMEM_LD_X16(tmem + lane_addr, rr);
    tc_wait_ld();
    for (int j = 0; j < 16; ++j) d[r * 16 + j] = __uint_as_float(rr[j]);
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        tmem_dealloc(tmem, 64);
    }
}

// probe: D[128, 128] = A[128, 64 k] * Bt[64 k, 128 n] with the B operand MN-major (n contiguous in memory, as the V rows
// of a KV cache are): Bt is staged as two 64-n atoms of [64 k rows][128 B], 128-byte swizzled -- the image a TMA box
// [64 n, 64 k rows] would leave -- and described with LBO = the atom stride along n, SBO = 1024 B between 8-row k groups
// (mode 2), or with the two swapped (mode 3: the reading that must NOT work).
__global__ void __launch_bounds__(128, 1)
probe_umma_mn_kernel(const __half* __restrict__ a, const __half* __restrict__ bt, float* __restrict__ d, int mode) {
    __shared__ __align__(1024) unsigned char s_a[128 * 128];
    __shared__ __align__(1024) unsigned char s_b[2 * 64 * 128];
    __shared__ uint64_t bar;
    __shared__ uint32_t s_tmem;
    const int warp = threadIdx.x >> 5, r = threadIdx.x;
    for (int c = 0; c < 8; ++c) {
        const uint4 va = *reinterpret_cast<const uint4*>(a + r * 64 + c * 8);
        *reinterpret_cast<uint4*>(s_a + (r >> 3) * 1024 + (r & 7) * 128 + ((c ^ (r & 7)) << 4)) = va;
    }
    for (int i = r; i < 2 * 64 * 8; i += 128) {                 // (atom, k row, 16-byte chunk)
        const int atom = i / (64 * 8), row = (i / 8) % 64, c = i % 8;
        const uint4 vb = *reinterpret_cast<const uint4*>(bt + row * 128 + atom * 64 + c * 8);
        *reinterpret_cast<uint4*>(s_b + atom * 8192 + (row >> 3) * 1024 + (row & 7) * 128 + ((c ^ (row & 7)) << 4)) = vb;
    }
    fence_proxy_async_smem();
    if (threadIdx.x == 0) {
        mbar_init(&bar, 1);
        fence_barrier_init();
    }
    if (warp == 0) {
        tmem_alloc(&s_tmem, 128);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = s_tmem;
    if (threadIdx.x == 0) {
        constexpr uint32_t idesc = umma_idesc_f16(128, 128) | (1u << 16);      // B MN-major
        const uint64_t lbo = mode == 2 ? 8192 : 1024, sbo = mode == 2 ? 1024 : 8192;
        for (int kk = 0; kk < 4; ++kk) {
            const uint64_t ad = umma_smem_desc_sw128(smem_u32(s_a) + kk * 32);
            uint64_t bd = 0;
            bd |= (uint64_t)(((smem_u32(s_b) + kk * 2048) & 0x3FFFF) >> 4);    // 16 k rows = two 8-row groups further
            bd |= (uint64_t)(lbo >> 4) << 16;
            bd |= (uint64_t)(sbo >> 4) << 32;
            bd |= (uint64_t)1 << 46;
            bd |= (uint64_t)2 << 61;
            umma_ss_f16(tmem, ad, bd, idesc, kk ? 1u : 0u);
        }
        umma_commit(&bar);
    }
    mbar_wait(&bar, 0);
    tc_fence_after();
    const uint32_t lane_addr = (uint32_t)(warp * 32) << 16;
    for (int c0 = 0; c0 < 128; c0 += 16) {
        uint32_t rr[16];
        UMB_TMEM_LD_X16(tmem + lane_addr + c0, rr);
        tc_wait_ld();
        for (int j = 0; j < 16; ++j) d[r * 128 + c0 + j] = __uint_as_float(rr[j]);
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        tmem_dealloc(tmem, 128);
    }
}

// ------------------------------------------------------------------------------------------------
// SIMT cross-check of the packed stream (tests only): one CTA per tile, thread = feature row.
// ------------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(128)
awq_gemm_simt_kernel(const unsigned char* __restrict__ packed, const __half* __restrict__ x, int64_t ldx,
                     __half* __restrict__ y, int64_t ldy, int M, int K, int N_total) {
    const int tile = blockIdx.x, r = threadIdx.x, G = K / kGroup;
    const int n = tile * kTileN + r;
    for (int m0 = 0; m0 < M; m0 += 8) {
        float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        for (int g = 0; g < G; ++g) {
            const unsigned char* rec = packed + ((int64_t)tile * G + g) * kRecordStride;
            const uint32_t zw = *reinterpret_cast<const uint32_t*>(rec + kRecZeroOff + (r >> 3) * 4);
            const int z = (int)((zw >> (4 * (r & 7))) & 0xFu);
            const __half s = *reinterpret_cast<const __half*>(rec + kRecScaleOff + r * 2);
            for (int c = 0; c < 4; ++c) {
                const uint4 w4 = *reinterpret_cast<const uint4*>(rec + (c * kTileN + r) * 16);
                const uint32_t words[4] = {w4.x, w4.y, w4.z, w4.w};
                for (int w = 0; w < 4; ++w)
                    for (int i = 0; i < 8; ++i) {
                        const float wf = __half2float(__hmul(__int2half_rn((int)((words[w] >> (4 * nib_pos(i))) & 0xFu) - z), s));
                        const int k = g * kGroup + c * 32 + w * 8 + i;
                        for (int j = 0; j < 8; ++j)
                            if (m0 + j < M) acc[j] = fmaf(__half2float(x[(int64_t)(m0 + j) * ldx + k]), wf, acc[j]);
                    }
            }
        }
        if (n < N_total)
            for (int j = 0; j < 8; ++j)
                if (m0 + j < M) y[(int64_t)(m0 + j) * ldy + n] = __float2half_rn(acc[j]);
    }
}

// ------------------------------------------------------------------------------------------------
// host side
// ------------------------------------------------------------------------------------------------
// fp16 row-major [rows, cols] (leading dimension ld elements) -> tiled map, box [64 cols, box_rows], SW128
static int make_tmap(CUtensorMap* map, const void* base, uint64_t rows, uint64_t cols, uint64_t ld, uint32_t box_rows) {
    PFN_encodeTiled enc = get_encode();
    if (!enc) return UMB_ERR_DRIVER;
    const cuuint64_t dims[2] = {cols, rows};
    const cuuint64_t strides[1] = {ld * sizeof(__half)};
    const cuuint32_t box[2] = {64, box_rows};
    const cuuint32_t estr[2] = {1, 1};
    const CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<void*>(base), dims, strides, box, estr,
                           CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                           CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return arg_fail(__FILE__, __LINE__, "cuTensorMapEncodeTiled");
    return UMB_OK;
}

// debug timeline (UMB_GEMM_TRACE=1): one device buffer, 16 stamps per CTA of the LAST gemm launch
static unsigned long long* trace_buffer() {
    static unsigned long long* buf = nullptr;
    static int tried = 0;
    if (!tried) {
        tried = 1;
        const char* e = getenv("UMB_GEMM_TRACE");
        if (e && e[0] == '1' && cudaMalloc(&buf, 1024 * 16 * sizeof(unsigned long long)) != cudaSuccess) buf = nullptr;
        if (buf) cudaMemset(buf, 0, 1024 * 16 * sizeof(unsigned long long));
    }
    return buf;
}

// UMB_GEMM_TRACE_LAUNCH=k: stamp only the k-th launch (0-based) after the last umb_debug_gemm_trace read, so that a
// launch in the middle of a back-to-back chain can be looked at without its neighbours overwriting the stamps
static int g_trace_launches = 0;
static unsigned long long* trace_for_this_launch() {
    unsigned long long* buf = trace_buffer();
    if (!buf) return nullptr;
    static int want = -2;
    if (want == -2) {
        const char* e = getenv("UMB_GEMM_TRACE_LAUNCH");
        want = e ? atoi(e) : -1;
    }
    const int idx = g_trace_launches++;
    return (want < 0 || idx == want) ? buf : nullptr;
}

static int mpad_of(int M) { return M <= 16 ? 16 : (M <= 32 ? 32 : (M <= 64 ? 64 : 128)); }

template <int MPAD, bool kAwq>
static int launch_gemm(const CUtensorMap& tx, const CUtensorMap& tw, GemmParams p, int grid, cudaStream_t st) {
    p.stages = kAwq ? GemmCfg<MPAD>::kStagesAwq : GemmCfg<MPAD>::kStagesF16;
    {
        static int env_stages = -1;
        if (env_stages < 0) {
            const char* e = getenv("UMB_GEMM_STAGES");
            env_stages = e ? atoi(e) : 0;
        }
        if (env_stages > 0 && env_stages <= 16 && (env_stages % 2) == 0 && !(kAwq && GemmCfg<MPAD>::kSplit) && GemmCfg<MPAD>::smem_bytes(kAwq, env_stages) <= 227 * 1024)
            p.stages = env_stages;                                   // even: see the static_assert on the ring depths
    }
    p.trace = trace_for_this_launch();
    const int smem = GemmCfg<MPAD>::smem_bytes(kAwq, p.stages);
    // per-device attribute (a process may drive several GPUs / threads): set on every launch, it is a cheap host call
    UMB_CUDA(cudaFuncSetAttribute(gemm_kernel<MPAD, kAwq>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    UMB_LAUNCH_PDL(gemm_kernel<MPAD, kAwq>, dim3(grid), dim3(kAwq ? GemmCfg<MPAD>::kThreadsAwq : kGemmThreadsF16), (size_t)smem, st, tx,
                   tw, p);
    count_launches(1);
    return UMB_OK;
}

static int gemm_common(bool awq, const void* x, int64_t ldx, const void* w, int64_t ldw, void* y, int64_t ldy, int M,
                       int K, int N_total, const umb_epilogue_t* epi, void* workspace, size_t workspace_bytes,
                       cudaStream_t st) {
    UMB_CHECK_ARG(x && w && y && M >= 1 && K >= 1 && N_total >= 1);
    UMB_CHECK_ARG((((uintptr_t)x | (uintptr_t)w) & 15) == 0 && (ldx % 8) == 0 && ldx >= K);
    if (const int gave_up = give_up_status()) return gave_up;
    if (M > (awq ? 512 : 128)) return UMB_ERR_UNSUPPORTED;
    if (awq ? (K % kGroup) != 0 : (K % 64) != 0) return UMB_ERR_UNSUPPORTED;
    if (N_total % 8) return UMB_ERR_UNSUPPORTED;
    GemmParams p{};
    p.packed = awq ? (const unsigned char*)w : nullptr;
    p.M = M;
    p.K = K;
    p.N_total = N_total;
    p.units_per_tile = awq ? K / kGroup : K / 64;
    p.tiles = (N_total + kTileN - 1) / kTileN;
    p.y = y;
    p.ldy = ldy;
    p.mode = epi ? epi->mode : UMB_EPI_STORE;
    p.bias = epi ? (const __half*)epi->bias : nullptr;
    p.residual = epi ? (const __half*)epi->residual : nullptr;
    p.ld_residual = epi ? epi->ld_residual : 0;
    p.argmax = epi ? epi->argmax : nullptr;

    UMB_CHECK_ARG(p.mode >= UMB_EPI_STORE && p.mode <= UMB_EPI_ROPE_QKV);
    if (p.mode == UMB_EPI_ROPE_QKV) {
        UMB_CHECK_ARG(epi->rope != nullptr);
        p.rope = *epi->rope;
        const umb_rope_epilogue_t& r = p.rope;
        UMB_CHECK_ARG(r.q_out && r.k_cache && r.v_cache && r.cos && r.sin && r.position_ids);
        UMB_CHECK_ARG((r.head_dim == 64 || r.head_dim == 128) && r.num_q_heads >= 1 && r.num_kv_heads >= 1);
        UMB_CHECK_ARG(N_total == (r.num_q_heads + 2 * r.num_kv_heads) * r.head_dim);
        const uintptr_t ptrs = (uintptr_t)r.q_out | (uintptr_t)r.k_cache | (uintptr_t)r.v_cache | (uintptr_t)r.cos | (uintptr_t)r.sin;
        p.rope_vec_ok = ((ptrs & 15) == 0 && (r.kv_tok_stride % 8) == 0 && (r.kv_head_stride % 8) == 0) ? 1 : 0;
    }
    if (p.mode == UMB_EPI_RESIDUAL) UMB_CHECK_ARG(p.residual != nullptr);
    p.vec_ok = (((uintptr_t)y & 15) == 0 && (ldy % 8) == 0 && (N_total % 8) == 0 &&
                (p.mode != UMB_EPI_RESIDUAL || ((((uintptr_t)p.residual) & 15) == 0 && (p.ld_residual % 8) == 0))) ? 1 : 0;
    if (p.mode == UMB_EPI_SILU_MUL) UMB_CHECK_ARG((N_total % kTileN) == 0 && p.bias == nullptr);

    if (awq && M > 128) {
        const size_t need = awq_wide_ws_bytes(M, N_total);
        if (!workspace || workspace_bytes < need) return UMB_ERR_WORKSPACE;
        UMB_CHECK_ARG(((uintptr_t)workspace & 15) == 0);
        if ((long long)(p.tiles + 1) * p.units_per_tile * 2 >= (1ll << 31)) return UMB_ERR_UNSUPPORTED;
        p.slots = reinterpret_cast<float*>(reinterpret_cast<unsigned char*>(workspace) + (((size_t)p.tiles * 4 + 255) & ~(size_t)255));
        return launch_awq_wide(x, ldx, p, st);
    }
    const int mpad = mpad_of(M);
    const long long U = (long long)p.tiles * p.units_per_tile;
    if (U >= (1ll << 31)) return UMB_ERR_UNSUPPORTED;
    int grid = sm_count();
    if ((long long)grid > U) grid = (int)U;
    static int aligned_split = -1;                   // UMB_GEMM_ALIGNED_SPLIT=0: plain stream-K for small problems too (tuning)
    if (aligned_split < 0) {
        const char* e = getenv("UMB_GEMM_ALIGNED_SPLIT");
        aligned_split = (e && e[0] == '0') ? 0 : 1;
    }
    if (aligned_split && U < 16ll * grid && p.tiles <= grid) {
        // small problem (draft-model linears): latency-bound, so cut every tile into the same power-of-two
        // number of k-slices (one segment per CTA, fewer partials per tile to reduce) instead of balancing units
        int S = 1;
        while (p.tiles * (S * 2) <= grid && p.units_per_tile % (S * 2) == 0) S *= 2;
        grid = p.tiles * S;
    }
    const size_t need = umb_gemm_workspace_bytes(M, K, N_total);
    if (!workspace || workspace_bytes < need) return UMB_ERR_WORKSPACE;
    UMB_CHECK_ARG(((uintptr_t)workspace & 15) == 0);
    p.counters = reinterpret_cast<int*>(workspace);
    p.slots = reinterpret_cast<float*>(reinterpret_cast<unsigned char*>(workspace) + (((size_t)p.tiles * 4 + 255) & ~(size_t)255));

    CUtensorMap tx, tw;
    int rc = make_tmap(&tx, x, (uint64_t)M, (uint64_t)K, (uint64_t)ldx, (uint32_t)mpad);
    if (rc != UMB_OK) return rc;
    if (!awq) {
        UMB_CHECK_ARG((ldw % 8) == 0 && ldw >= K);
        rc = make_tmap(&tw, w, (uint64_t)N_total, (uint64_t)K, (uint64_t)ldw, (uint32_t)kTileN);
        if (rc != UMB_OK) return rc;
    } else {
        rc = make_tmap_x3d(&tw, x, (uint64_t)M, (uint64_t)K, (uint64_t)ldx, (uint32_t)mpad);   // AWQ: tmap_w = x as slabs
        if (rc != UMB_OK) return rc;
    }
    if (sync_debug())
        fprintf(stderr, "umbrella_b200: gemm awq=%d M=%d K=%d N=%d mode=%d grid=%d mpad=%d\n", (int)awq, M, K, N_total, p.mode,
                grid, mpad);
#define UMB_DISPATCH(MP)                                                       \
    return awq ? launch_gemm<MP, true>(tx, tw, p, grid, st) : launch_gemm<MP, false>(tx, tw, p, grid, st)
    switch (mpad) {
        case 16: UMB_DISPATCH(16);
        case 32: UMB_DISPATCH(32);
        case 64: UMB_DISPATCH(64);
        default: UMB_DISPATCH(128);
    }
#undef UMB_DISPATCH
}

// The pair kernel sums a tile's k in one accumulator, the kernel of up to 128 rows in two, and has twice the k of a tile to a block; the tensor core cuts a sum
// off at every step.  Distance to float64 of fp16 results, 300 to 512 rows, passes of up to 128 rows / pairs: K = 4096 2.0732e-4 / 2.0735e-4 (28672 features), 8192 + 0.04 to
// 0.05 %, 14336 + 0.045 %, 28672 2.072e-4 / 2.083e-4, for 10 % of the time (28672 -> 8192, 500 rows, us: 218 / 193; 300 rows 149 / 170).  So the longest go in passes.
constexpr int kWideK = 16384;
int awq_gemm_rows(const void* x, int64_t ldx, const void* packed, void* y, int64_t ldy, int M, int K, int N_total, const umb_epilogue_t* epi,
                  void* workspace, size_t workspace_bytes, cudaStream_t st) {
    const int mode = epi ? epi->mode : UMB_EPI_STORE;
    if (M <= 128 || M > 512 || K <= kWideK || mode == UMB_EPI_ROPE_QKV)
        return gemm_common(true, x, ldx, packed, 0, y, ldy, M, K, N_total, epi, workspace, workspace_bytes, st);
    const int passes = (M + 127) / 128, rows = (M + passes - 1) / passes;
    for (int r0 = 0; r0 < M; r0 += rows) {
        umb_epilogue_t e{};
        if (epi) e = *epi;
        if (e.residual) e.residual = (const __half*)e.residual + (int64_t)r0 * e.ld_residual;
        if (e.argmax) e.argmax += r0;
        const size_t size = mode == UMB_EPI_LOGITS ? sizeof(float) : sizeof(__half);
        const int rc = gemm_common(true, (const __half*)x + (int64_t)r0 * ldx, ldx, packed, 0, (unsigned char*)y + (int64_t)r0 * ldy * size, ldy, M - r0 < rows ? M - r0 : rows, K,
                                   N_total, epi ? &e : nullptr, workspace, workspace_bytes, st);
        if (rc != UMB_OK) return rc;
    }
    return UMB_OK;
}

}  // namespace umb

using namespace umb;

extern "C" size_t umb_awq_packed_bytes(int K, int N_total, int group) {
    if (group != kGroup || K <= 0 || N_total <= 0 || (K % kGroup) != 0) return 0;
    return (size_t)((N_total + kTileN - 1) / kTileN) * (K / kGroup) * kRecordStride;
}

extern "C" size_t umb_gemm_workspace_bytes(int M, int K, int N_total) {
    (void)K;
    if (M < 1 || N_total < 1) return 0;
    const size_t tiles = (size_t)(N_total + kTileN - 1) / kTileN;
    const size_t mpad = (size_t)mpad_of(M > 128 ? 128 : M);
    const size_t slots = tiles + 1024;   // tiles + an upper bound on the grid size
    return ((tiles * 4 + 255) & ~(size_t)255) + slots * mpad * kTileN * sizeof(float);
}

extern "C" int umb_awq_repack(const int32_t* qweight, const int32_t* qzeros, const void* scales, int K, int N, int group,
                              void* packed, int N_total, int row_block, int row_stride, int row_offset,
                              umb_stream_t stream) {
    UMB_CHECK_ARG(qweight && qzeros && scales && packed);
    if (group != kGroup) return UMB_ERR_UNSUPPORTED;
    UMB_CHECK_ARG(K > 0 && N > 0 && (K % kGroup) == 0 && (N % 8) == 0);
    UMB_CHECK_ARG(row_block > 0 && (row_block % 8) == 0 && (row_offset % 8) == 0 && (row_stride % 8) == 0);
    UMB_CHECK_ARG((N % row_block) == 0 || N < row_block);
    const int64_t last = (int64_t)((N - 1) / row_block) * row_stride + row_offset + (N - 1) % row_block;
    UMB_CHECK_ARG(last < (int64_t)((N_total + kTileN - 1) / kTileN) * kTileN);
    cudaStream_t st = (cudaStream_t)stream;
    const int cols = N / 8;
    awq_repack_weights_kernel<<<dim3((cols + 127) / 128, K / 8), 128, 0, st>>>(qweight, K, N, (unsigned char*)packed,
                                                                                row_block, row_stride, row_offset);
    awq_repack_meta_kernel<<<dim3((cols + 127) / 128, K / kGroup), 128, 0, st>>>(
        qzeros, (const __half*)scales, K, N, (unsigned char*)packed, row_block, row_stride, row_offset);
    count_launches(2);
    UMB_LAUNCH_CHECK();
    return UMB_OK;
}

extern "C" int umb_awq_dequantize_f16(const int32_t* qweight, const int32_t* qzeros, const void* scales, int K, int N,
                                      int group, void* out, umb_stream_t stream) {
    UMB_CHECK_ARG(qweight && qzeros && scales && out);
    if (group != kGroup) return UMB_ERR_UNSUPPORTED;
    UMB_CHECK_ARG(K > 0 && N > 0 && (K % kGroup) == 0 && (N % 8) == 0);
    awq_dequantize_kernel<<<dim3((N / 8 + 127) / 128, K), 128, 0, (cudaStream_t)stream>>>(
        qweight, qzeros, (const __half*)scales, K, N, (__half*)out);
    count_launches(1);
    UMB_LAUNCH_CHECK();
    return UMB_OK;
}

extern "C" int umb_awq_unpack_f16(const void* packed, int K, int N_total, int group, void* out, umb_stream_t stream) {
    UMB_CHECK_ARG(packed && out);
    if (group != kGroup) return UMB_ERR_UNSUPPORTED;
    UMB_CHECK_ARG(K > 0 && N_total > 0 && (K % kGroup) == 0);
    awq_unpack_kernel<<<dim3((K / 8 + 127) / 128, N_total), 128, 0, (cudaStream_t)stream>>>(
        (const unsigned char*)packed, K, N_total, (__half*)out);
    count_launches(1);
    UMB_LAUNCH_CHECK();
    return UMB_OK;
}

extern "C" int umb_awq_gemm_f16(const void* x, int64_t ldx, const void* packed, void* y, int64_t ldy, int M, int K,
                                int N_total, int group, const umb_epilogue_t* epilogue, void* workspace,
                                size_t workspace_bytes, umb_stream_t stream) {
    if (group != kGroup || M > 128) return UMB_ERR_UNSUPPORTED;
    return gemm_common(true, x, ldx, packed, 0, y, ldy, M, K, N_total, epilogue, workspace, workspace_bytes,
                       (cudaStream_t)stream);
}

extern "C" size_t umb_awq_gemm_rows_ws_bytes(int M, int K, int N_total) {
    if (M < 1 || M > 512 || N_total < 1) return 0;
    const size_t few = umb_gemm_workspace_bytes(M, K, N_total), many = M > 128 ? awq_wide_ws_bytes(M, N_total) : 0;
    return few > many ? few : many;
}

extern "C" int umb_awq_gemm_rows_f16(const void* x, int64_t ldx, const void* packed, void* y, int64_t ldy, int M, int K,
                                     int N_total, int group, const umb_epilogue_t* epilogue, void* workspace,
                                     size_t workspace_bytes, umb_stream_t stream) {
    if (group != kGroup) return UMB_ERR_UNSUPPORTED;
    return awq_gemm_rows(x, ldx, packed, y, ldy, M, K, N_total, epilogue, workspace, workspace_bytes, (cudaStream_t)stream);
}

extern "C" int umb_gemm_f16(const void* x, int64_t ldx, const void* w, int64_t ldw, void* y, int64_t ldy, int M, int K,
                            int N, const umb_epilogue_t* epilogue, void* workspace, size_t workspace_bytes,
                            umb_stream_t stream) {
    return gemm_common(false, x, ldx, w, ldw, y, ldy, M, K, N, epilogue, workspace, workspace_bytes,
                       (cudaStream_t)stream);
}

extern "C" int umb_debug_gemm_trace(unsigned long long* host_out, int max_ctas) {
    unsigned long long* buf = trace_buffer();
    if (!buf || !host_out || max_ctas < 1) return UMB_ERR_ARG;
    if (max_ctas > 1024) max_ctas = 1024;
    UMB_CUDA(cudaDeviceSynchronize());
    UMB_CUDA(cudaMemcpy(host_out, buf, (size_t)max_ctas * 16 * sizeof(unsigned long long), cudaMemcpyDeviceToHost));
    UMB_CUDA(cudaMemset(buf, 0, 1024 * 16 * sizeof(unsigned long long)));
    g_trace_launches = 0;
    return UMB_OK;
}

extern "C" int umb_probe_umma(const void* a, const void* b, float* d, int mode, umb_stream_t stream) {
    UMB_CHECK_ARG(a && b && d && mode >= 0 && mode <= 3);
    if (mode >= 2)      // B operand MN-major: b is fp16 [64 k, 128 n], d fp32 [128, 128]
        probe_umma_mn_kernel<<<1, 128, 0, (cudaStream_t)stream>>>((const __half*)a, (const __half*)b, d, mode);
    else
        probe_umma_kernel<<<1, 128, 0, (cudaStream_t)stream>>>((const __half*)a, (const __half*)b, d, mode);
    count_launches(1);
    UMB_LAUNCH_CHECK();
    return UMB_OK;
}

extern "C" int umb_awq_gemm_f16_simt(const void* x, int64_t ldx, const void* packed, void* y, int64_t ldy, int M, int K,
                                     int N_total, umb_stream_t stream) {
    UMB_CHECK_ARG(x && packed && y && M >= 1 && K > 0 && (K % kGroup) == 0 && N_total > 0);
    awq_gemm_simt_kernel<<<(N_total + kTileN - 1) / kTileN, 128, 0, (cudaStream_t)stream>>>(
        (const unsigned char*)packed, (const __half*)x, ldx, (__half*)y, ldy, M, K, N_total);
    count_launches(1);
    UMB_LAUNCH_CHECK();
    return UMB_OK;
}
