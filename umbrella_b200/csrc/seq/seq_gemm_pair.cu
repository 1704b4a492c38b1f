// Dense products of many rows, tiles of 256 rows x 256 columns by pairs of SMs (tcgen05 cta_group::2): a block of the pair holds 128 rows
// of activations and 128 of the tile's 256 weight rows, and the tensor cores of both read the two halves of the weights.  What a block
// brings in and reads for a step of 64 of k falls from 48 KB to 32 KB, which is what bounds a block on its own: 96 KB in and out of shared
// memory per 512 clocks of products (seq_gemm_tc.cu, 690 clocks a step).
//
// Both blocks run the same roles: warp 0 copies its halves with TMA, counted by the first block's barrier; warp 1 of the first block
// issues the products and tells both blocks when a stage is free and a tile done; warps 2-9 store the block's own 128 rows, half of
// the columns each four (with four warps, 1024 of k are over before 128 x 256 results are stored).
#include "seq_gemm_walk.cuh"

namespace umbs {

constexpr int kPrStages = 5, kPrStage = 2 * kTcRows * 128;  // 128 rows of activations, 128 of weights
constexpr int kPrStore = 8, kPrThreads = 64 + 32 * kPrStore;        // warps that store
constexpr int kPrSmem = 1024 + kPrStages * kPrStage + kPrStore * 32 * kTcStageRow * 4;

__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_sync() { asm volatile("barrier.cluster.arrive.aligned;\n\tbarrier.cluster.wait.aligned;" ::: "memory"); }
// the address of the first block's barrier, for both
__device__ __forceinline__ uint32_t first_block(const void* p) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(r) : "r"(smem_u32(p)));
    return r;
}
__device__ __forceinline__ void arrive_at(uint32_t bar) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tma_3d_pair(void* dst, const CUtensorMap* map, int c0, int c1, int c2, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
                 ::"r"(smem_u32(dst)), "l"(map), "r"(c0), "r"(c1), "r"(c2), "r"(bar) : "memory");
}
__device__ __forceinline__ void umma_pair(uint32_t d, uint64_t ad, uint64_t bd, uint32_t idesc, uint32_t accumulate) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
                 ::"r"(d), "l"(ad), "l"(bd), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void commit_pair(uint64_t* bar) {               // the same barrier of both blocks
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
                 ::"r"(smem_u32(bar)), "h"((uint16_t)3) : "memory");
}
// waits on barriers that the other block arrives at
__device__ __forceinline__ bool spin_pair(uint64_t* bar, uint32_t parity, volatile int* quit) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t.reg .u32 n;\n\tmov.u32 n, 0;\n\t"
        "AGAIN_%=:\n\t"
        "mbarrier.test_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "@p bra DONE_%=;\n\t"
        "add.u32 n, n, 1;\n\tsetp.lt.u32 q, n, 33554432;\n\t@q bra AGAIN_%=;\n\t"
        "DONE_%=:\n\tselp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity) : "memory");
    return __all_sync(0xffffffffu, ok) || tc_give_up(quit);
}

template <bool DUAL, typename TC>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kPrThreads, 1)
gemm_pair_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_w, const __grid_constant__ GemmArgs a, const __grid_constant__ TcArgs t) {
    constexpr int kOut = DUAL ? 128 : 256;                  // output columns of a tile
    extern __shared__ unsigned char smem_raw[];
    __shared__ uint64_t bars[2 * kPrStages + 4];
    __shared__ uint32_t s_tmem;
    __shared__ int s_quit;
    unsigned char* smem = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    float* s_out = reinterpret_cast<float*>(smem + kPrStages * kPrStage);
    uint64_t *full = bars, *empty = bars + kPrStages, *acc_full = bars + 2 * kPrStages, *acc_empty = acc_full + 2;
    volatile int* quit = &s_quit;
    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
    const uint32_t rank = cluster_rank();
    if (threadIdx.x == 0) {
        umb::tma_prefetch_desc(&map_w);
        umb::tma_prefetch_desc(&map_a);
        for (int i = 0; i < kPrStages; ++i) {
            umb::mbar_init(full + i, 1);
            umb::mbar_init(empty + i, 1);
        }
        for (int i = 0; i < 2; ++i) {
            umb::mbar_init(acc_full + i, 1);
            umb::mbar_init(acc_empty + i, 2 * kPrStore);
        }
        s_quit = 0;
        umb::fence_barrier_init();
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(&s_tmem)) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;");
    }
    umb::tc_fence_before();
    __syncthreads();
    cluster_sync();                                         // both blocks' barriers are there
    umb::tc_fence_after();
    const uint32_t tmem = s_tmem;
    chain_wait();

    // the pair's tiles: rows fastest, then columns, then groups
    const int per_group = t.m_tiles * t.n_tiles, tiles = t.groups * per_group, pairs = gridDim.x >> 1;
    if (warp == 0) {
        uint32_t s = 0, ph = 1;
        bool ok = true, ready = false;
        for (int i = blockIdx.x >> 1; ok && i < tiles; i += pairs) {
            const int g = i / per_group, j = i - g * per_group, n0 = j / t.m_tiles, m0 = (j - n0 * t.m_tiles) * 256 + (int)rank * 128;
            const int gw = t.w_grouped ? g : 0, ga = t.a_grouped ? g : 0;
            const int wr = DUAL ? (int)rank * a.N + n0 * 128 : n0 * 256 + (int)rank * 128;      // (DUAL: gate rows in the first block, up rows in the second)
            for (int k = 0; k < t.k_steps; ++k) {
                if (!ready && !(ok = spin_pair(empty + s, ph, quit))) break;
                unsigned char* st = smem + s * kPrStage;
                const uint32_t bar = first_block(full + s), s2 = s + 1 == kPrStages ? 0 : s + 1, ph2 = s + 1 == kPrStages ? ph ^ 1 : ph;
                const bool next = tc_test(empty + s2, ph2);
                if (umb::elect_one()) {
                    if (rank == 0) umb::mbar_arrive_expect_tx(full + s, 2 * kPrStage);
                    tma_3d_pair(st, &map_a, k * kTcK, m0, ga, bar);
                    tma_3d_pair(st + kTcRows * 128, &map_w, k * kTcK, wr, gw, bar);
                }
                ready = __all_sync(0xffffffffu, next);
                s = s2;
                ph = ph2;
            }
        }
    } else if (warp == 1) {
        if (rank == 0) {
            constexpr uint32_t idesc = tc_idesc(256, 256);
            uint32_t s = 0, ph = 0, it = 0;
            bool ok = true, ready = false;
            for (int i = blockIdx.x >> 1; ok && i < tiles; i += pairs, ++it) {
                const uint32_t acc = it & 1, d = tmem + acc * 256;
                if (!(ok = spin_pair(acc_empty + acc, ((it >> 1) & 1) ^ 1, quit))) break;
                umb::tc_fence_after();
                for (int k = 0; k < t.k_steps; ++k) {
                    if (!ready && !(ok = spin_pair(full + s, ph, quit))) break;
                    const uint32_t s2 = s + 1 == kPrStages ? 0 : s + 1, ph2 = s + 1 == kPrStages ? ph ^ 1 : ph;
                    const bool next = tc_test(full + s2, ph2);
                    umb::tc_fence_after();
                    const uint32_t st = smem_u32(smem + s * kPrStage);
                    const uint64_t ad = umb::umma_smem_desc_sw128(st), wd = umb::umma_smem_desc_sw128(st + kTcRows * 128);
                    if (umb::elect_one()) {
#pragma unroll
                        for (int kk = 0; kk < kTcK / 16; ++kk) umma_pair(d, ad + kk * 2, wd + kk * 2, idesc, (k | kk) ? 1u : 0u);
                        commit_pair(empty + s);
                        if (k + 1 == t.k_steps) commit_pair(acc_full + acc);
                    }
                    ready = __all_sync(0xffffffffu, next);
                    s = s2;
                    ph = ph2;
                }
            }
        }
    } else {
        const int q = warp & 3, half = (warp - 2) >> 2 ? kOut / 2 : 0;        // half of the columns
        float* so = s_out + (warp - 2) * 32 * kTcStageRow;
        uint32_t it = 0;
        for (int i = blockIdx.x >> 1; i < tiles; i += pairs, ++it) {
            const int g = i / per_group, j = i - g * per_group, n0 = j / t.m_tiles, row = (j - n0 * t.m_tiles) * 256 + (int)rank * 128 + q * 32;
            const uint32_t acc = it & 1;
            if (!__all_sync(0xffffffffu, tc_poll(acc_full + acc, (it >> 1) & 1, quit))) break;
            umb::tc_fence_after();
            tc_store_tile<kOut / 2, kOut, DUAL, TC>(a, t.vec_c, tmem + acc * 256 + half + ((uint32_t)(q * 32) << 16), so, g, row, a.M - row,
                                                    n0 * kOut + half, [&] { arrive_at(first_block(acc_empty + acc)); });
        }
    }
    __syncwarp();
    umb::tc_fence_before();
    __syncthreads();
    tc_settle(quit, t.report);
    cluster_sync();                                         // neither block's memory goes while the other's products or copies use it
    if (warp == 1) {
        umb::tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, 512;" ::"r"(tmem));
    }
}

template <bool DUAL, typename TC>
static int launch_pair(const GemmArgs& a, TcArgs t, int sms, cudaStream_t st) {
    constexpr int out = DUAL ? 128 : 256;
    t.n_tiles = (a.N + out - 1) / out;
    t.m_tiles = (a.M + 255) / 256;
    t.k_steps = (a.K + kTcK - 1) / kTcK;
    const int ga = a.a_goff != 0 ? t.groups : 1, gw = a.w_gstride != 0 ? t.groups : 1;
    t.a_grouped = ga > 1;
    t.w_grouped = gw > 1;
    CUtensorMap ma{}, mw{};
    int rc = encode_map(&mw, a.W, a.K, (uint64_t)a.N * (DUAL ? 2 : 1), gw, a.ldw, a.w_gstride, 128);
    if (rc == 0) rc = encode_map(&ma, a.A, a.K, a.M, ga, a.lda, a.a_goff, kTcRows);
    if (rc != 0) return rc;
    auto kernel = gemm_pair_kernel<DUAL, TC>;
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kPrSmem);
    if (e != cudaSuccess) return (int)e;
    const int64_t tiles = (int64_t)t.groups * t.m_tiles * t.n_tiles;
    return chain_launch(kernel, 2 * (int)(tiles < sms / 2 ? tiles : sms / 2), kPrThreads, kPrSmem, st, ma, mw, a, t);
}

int launch_gemm_pair(const GemmArgs& a, TcArgs t, bool dual, bool c_f32, int sms, cudaStream_t st) {
    if (dual) return c_f32 ? launch_pair<true, float>(a, t, sms, st) : launch_pair<true, __nv_bfloat16>(a, t, sms, st);
    return c_f32 ? launch_pair<false, float>(a, t, sms, st) : launch_pair<false, __nv_bfloat16>(a, t, sms, st);
}

unsigned int pair_timeouts() { return tc_timeouts(); }

}  // namespace umbs
