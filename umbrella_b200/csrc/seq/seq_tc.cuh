// Bounded mbarrier waits of the tensor-core kernels of the sequence-state decoders.
#pragma once
#include <cuda.h>

#include "../common.cuh"
#include "seq_internal.h"

namespace umbs {
using umb::smem_u32;

static __device__ unsigned int g_tc_timeouts;               // blocks of this file's kernels that gave up on a wait

// Every wait is bounded (about a second): a block that gives up raises its flag, and every role of it leaves its loop.
__device__ __forceinline__ bool tc_give_up(volatile int* quit) {
    if (!*quit) {
        *quit = 1;
        atomicAdd(&g_tc_timeouts, 1u);
    }
    return false;
}
__device__ __forceinline__ bool tc_test(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity) : "memory");
    return ok != 0;
}
// Polling by a whole warp on a critical path (a parked thread comes back about a microsecond later); it is one again behind it (the loop as one statement: as C++ its exits cost 100 clocks a wait).  The warps that issue copies and products run their loops whole and
// elect a thread for the instructions themselves: inside a branch that one thread takes, operands leave the uniform registers
// and every tcgen05 instruction and every passed wait costs hundreds of clocks (measured with clock64 stamps: 8 products of
// 128 x 32 x 16 and a passed wait 1740 clocks, a wait for a finished barrier 370).
__device__ __forceinline__ bool tc_spin_for(uint64_t* bar, uint32_t parity) {      // false: time is up
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t.reg .u32 n;\n\tmov.u32 n, 0;\n\t"
        "AGAIN_%=:\n\t"
        "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "@p bra DONE_%=;\n\t"
        "add.u32 n, n, 1;\n\tsetp.lt.u32 q, n, 33554432;\n\t@q bra AGAIN_%=;\n\t"
        "DONE_%=:\n\tselp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity) : "memory");
    return __all_sync(0xffffffffu, ok);
}
__device__ __forceinline__ bool tc_spin_warp(uint64_t* bar, uint32_t parity, volatile int* quit) { return tc_spin_for(bar, parity) || tc_give_up(quit); }
// polling with a short sleep in between: for warps that share a scheduler with working ones
__device__ __forceinline__ bool tc_poll_for(uint64_t* bar, uint32_t parity, volatile int* quit) {        // false: time is up, or another role gave up
    for (int i = 0; i < (1 << 24); ++i) {
        if (tc_test(bar, parity)) return true;
        __nanosleep(20);
        if ((i & 255) == 255 && *quit) return false;
    }
    return false;
}
__device__ __forceinline__ bool tc_poll(uint64_t* bar, uint32_t parity, volatile int* quit) { return tc_poll_for(bar, parity, quit) || tc_give_up(quit); }
// Behind the last barrier of a kernel that gave up: the host learns of it (give_up_word), and copies and products in flight end
// before their memory goes.
__device__ __forceinline__ void tc_settle(volatile int* quit, volatile unsigned int* report) {
    if (!*quit) return;
    if (threadIdx.x == 0) {
        *report = 1u;
        __threadfence_system();
    }
    for (int i = 0; i < 1000; ++i) __nanosleep(1000);
    __syncthreads();
}

__host__ __device__ constexpr uint32_t tc_idesc(uint32_t M, uint32_t N, bool w_mn_major = false) {   // kind::f16, bf16 x bf16 -> fp32
    return (1u << 4) | (1u << 7) | (1u << 10) | ((w_mn_major ? 1u : 0u) << 16) | ((N >> 3) << 17) | ((M >> 4) << 24);
}

// The sigmoids' quotient without the rounded division's branch, which costs 12 us of 50 over 4096 rows of 2 x 2048 sums: the
// hardware's approximate reciprocal and one Newton-Raphson step, r (2 - x r) with the residual in one rounding: the rounded quotient for every x
// below 2^126 (all 1.06e9 compared).  Behind that the quotient is below the smallest normal number and becomes 0.
__device__ __forceinline__ float tc_sigmoid(float z) {
    const float x = 1.f + expf(-z), r = __fdividef(1.f, x);
    return x >= 0x1p126f ? 0.f : fmaf(r, fmaf(-x, r, 1.f), r);
}
// Eight fp32 numbers times 2^24 (SCALED: they are that already) as three rows of eight bf16, rounded to nearest one after the other: their sum, exactly, for all numbers up
// to 2^103.  (bf16 has fp32's range, so the parts of an fp32 number below 2^-110 would end below bf16's smallest, 2^-133; scaled,
// the lowest bit of the smallest subnormal is 2^-125, a normal number.)  Numbers beyond are infinite or NaN in their parts, and so are the sums
// they enter.  A product of two such operands is 2^48 times the operands': kSplitBack takes it back, exactly where the result is normal.
constexpr float kSplitScale = 0x1p24f, kSplitBack = 0x1p-48f;
template <bool SCALED = false>
__device__ __forceinline__ void split8(const float (&f)[8], uint4 (&p)[3]) {
    uint32_t* o[3] = {&p[0].x, &p[1].x, &p[2].x};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        float a = SCALED ? f[2 * i] : f[2 * i] * kSplitScale, b = SCALED ? f[2 * i + 1] : f[2 * i + 1] * kSplitScale;
#pragma unroll
        for (int e = 0; e < 3; ++e) {
            const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
            const uint32_t u = *reinterpret_cast<const uint32_t*>(&h);
            o[e][i] = u;
            a -= __uint_as_float(u << 16);
            b -= __uint_as_float(u & 0xffff0000u);
        }
    }
}

static inline unsigned int tc_timeouts() {
    unsigned int n = 0;
    return cudaMemcpyFromSymbol(&n, g_tc_timeouts, sizeof n) == cudaSuccess ? n : ~0u;
}
unsigned int attention_tc_timeouts();                       // seq_attn_tc.cu
unsigned int split_timeouts();                              // seq_gemm_split.cu
unsigned int chunk_tc_timeouts();                           // seq_chunk_tc.cu
unsigned int pair_timeouts();                               // seq_gemm_pair.cu

// seq_gemm_tc.cu: bf16 [groups][rows][cols] with row stride ld and group stride gs (elements) as a tensor map of boxes of 64
// columns x box_rows rows, 128-byte swizzle, zeros outside
int encode_map(CUtensorMap* map, const void* base, uint64_t cols, uint64_t rows, uint64_t groups, uint64_t ld, uint64_t gs, uint32_t box_rows);

__device__ __forceinline__ void tma_3d(void* dst, const CUtensorMap* map, int c0, int c1, int c2, uint64_t* bar) {
    asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
                 ::"r"(smem_u32(dst)), "l"(map), "r"(c0), "r"(c1), "r"(c2), "r"(smem_u32(bar)) : "memory");
}

}  // namespace umbs
