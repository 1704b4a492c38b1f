// Matrix products of steps with more than a few rows on the 5th-generation tensor cores: C = A W^T, bf16 operands, fp32 sums
// in tensor memory.
//
// A persistent block per SM walks output tiles of 128 rows x BN columns.  Warp 0 copies weight tiles (and, for dense rows,
// activation tiles) with TMA into a ring of 64-wide k steps, one thread of warp 1 issues tcgen05.mma, four or eight more empty the
// accumulators -- two sets of them, so that a tile is stored while the next one is summed.  Rows that are gathered or sorted by
// expert come from four to eight more warps through 16-byte cp.async: which rows a tile has is known on the device alone, and a tile
// of few rows fetches only those.
//
// An output element is one fp32 sum over k in the same order whatever its tile's size, so a row's result does not depend on
// the rest of the batch; against float64 it is as far off as the mma.sync tiles that this replaced (2.1e-6 at K = 2048, in
// both the tensor core's own accumulation).
//
// Bound for dense prompts: a block's shared memory, 48 KB in and 48 KB out for 512 clocks of products at 256 columns (690 clocks a step); the
// large ones go to pairs of SMs (seq_gemm_pair.cu).  With few steps: launch, first operands, last results (8.0 us for K = 1024 to 1024
// columns, 3.8 of them steps).  Sorted rows: the copying warps' loads (890 clocks a step of gathered ones; leaving them out: 7 us of 193) and the results
// (25 us of 193 with four warps that store).  16 experts, top 2, of width 2048 with the routing around it, us, four warps that store / eight:
// 64 tokens 85 / 73, 4096 210 / 208; gate|up of 64 tokens reads its 134 MB at the memory's rate.
// (tile::gather4 for tiles of few rows and boxes for full ones, with maps that went on behind the rows' memory, gave no more, and one run of them ended with an
// illegal address.)
#include <cuda.h>
#include <atomic>
#include <mutex>

#include "seq_gemm_walk.cuh"

namespace umbs {

template <int BN, bool DUAL>
struct TcCfg {
    static constexpr int kStages = BN == 256 ? 4 : (BN == 128 ? 6 : 8);
    // Rows copied by threads: every stage of the ring has its own warps, which fill it, wait for their copies and publish it.
    // (Warps that serve the stages in turn publish one only when they come back for another: 1.5 us per k step, a round trip
    // between the tensor core and the copies.)
    static constexpr int kWarpsPerStage = BN == 256 ? 2 : 1, kCopyWarps = kStages * kWarpsPerStage;
    // Warps that store: at 256 columns eight, half of the columns each four, 16 at a time (their staging blocks fit beside four stages).
    static constexpr int kStore = BN == 256 ? 8 : 4, kStoreCols = BN == 256 ? 16 : 32, kStoreBlock = 32 * (kStoreCols + 4);
    static constexpr int threads(bool dense) { return 64 + 32 * kStore + (dense ? 0 : 32 * kCopyWarps); }
    static constexpr int kABytes = kTcRows * 128, kWBytes = BN * 128, kStage = kABytes + kWBytes;
    static constexpr int kOut = DUAL ? BN / 2 : BN;         // output columns of a tile
    static constexpr int kSmem = 1024 + kStages * kStage + kStore * kStoreBlock * 4 + 256 + kCopyWarps * kTcRows * 4;
};

template <int BN, bool DUAL, bool DENSE, typename TC>
__global__ void __launch_bounds__(TcCfg<BN, DUAL>::threads(DENSE), 1)
gemm_tc_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_w, const GemmArgs a, const TcArgs t) {
    using Cfg = TcCfg<BN, DUAL>;
    constexpr int kStages = Cfg::kStages, kOut = Cfg::kOut;
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    float* s_out = reinterpret_cast<float*>(smem + kStages * Cfg::kStage);
    uint64_t* bars = reinterpret_cast<uint64_t*>(s_out + Cfg::kStore * Cfg::kStoreBlock);
    uint64_t *full = bars, *empty = bars + kStages, *acc_full = bars + 2 * kStages, *acc_empty = acc_full + 2;
    uint32_t* s_tmem = reinterpret_cast<uint32_t*>(acc_empty + 2);
    volatile int* quit = reinterpret_cast<volatile int*>(s_tmem + 1);
    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;

    if (threadIdx.x == 0) {
        umb::tma_prefetch_desc(&map_w);
        if (DENSE) umb::tma_prefetch_desc(&map_a);
        for (int i = 0; i < kStages; ++i) {
            umb::mbar_init(full + i, DENSE ? 1 : 1 + Cfg::kWarpsPerStage);         // the TMA thread and the stage's copying warps
            umb::mbar_init(empty + i, 1);
        }
        for (int i = 0; i < 2; ++i) {
            umb::mbar_init(acc_full + i, 1);
            umb::mbar_init(acc_empty + i, Cfg::kStore);
        }
        *quit = 0;
        umb::fence_barrier_init();
    }
    if (warp == 1) {
        umb::tmem_alloc(s_tmem, 2 * BN);
        umb::tmem_relinquish();
    }
    umb::tc_fence_before();
    __syncthreads();
    umb::tc_fence_after();
    const uint32_t tmem = *s_tmem;
    chain_wait();
    TileWalk w(a, t);

    if (warp == 0) {
        uint32_t s = 0, ph = 1;
        bool ok = true, ready = false;
        while (ok && w.step()) {
            const int gw = t.w_grouped ? w.g : 0, ga = t.a_grouped ? w.g : 0, n0 = w.n0 * kOut;
            for (int k = 0; k < t.k_steps; ++k) {
                if (!ready && !(ok = tc_spin_warp(empty + s, ph, quit))) break;
                unsigned char* st = smem + s * Cfg::kStage;
                const uint32_t s2 = s + 1 == kStages ? 0 : s + 1, ph2 = s + 1 == kStages ? ph ^ 1 : ph;
                const bool next = tc_test(empty + s2, ph2);             // (known behind the copies: no wait of its own where it is free)
                if (umb::elect_one()) {
                    umb::mbar_arrive_expect_tx(full + s, (DENSE ? Cfg::kABytes : 0) + Cfg::kWBytes);
                    if (DENSE) tma_3d(st, &map_a, k * kTcK, w.m0, ga, full + s);
                    tma_3d(st + Cfg::kABytes, &map_w, k * kTcK, n0, gw, full + s);
                    if (DUAL) tma_3d(st + Cfg::kABytes + kOut * 128, &map_w, k * kTcK, a.N + n0, gw, full + s);
                }
                ready = __all_sync(0xffffffffu, next);
                s = s2;
                ph = ph2;
            }
        }
    } else if (warp == 1) {
        constexpr uint32_t idesc = tc_idesc(kTcRows, BN);
        // Whether the next step's operands are there is asked in front of this step's products and known behind them: a wait for a
        // barrier that is through costs 300 clocks, and the tensor core has no more than two products in hand.
        uint32_t s = 0, ph = 0, it = 0;
        bool ok = true, ready = false;
        for (; ok && w.step(); ++it) {
            const uint32_t acc = it & 1, d = tmem + acc * BN;
            if (!(ok = tc_spin_warp(acc_empty + acc, ((it >> 1) & 1) ^ 1, quit))) break;
            umb::tc_fence_after();
            for (int k = 0; k < t.k_steps; ++k) {
                if (!ready && !(ok = tc_spin_warp(full + s, ph, quit))) break;
                const uint32_t s2 = s + 1 == kStages ? 0 : s + 1, ph2 = s + 1 == kStages ? ph ^ 1 : ph;
                const bool next = tc_test(full + s2, ph2);
                umb::tc_fence_after();
                const uint32_t st = smem_u32(smem + s * Cfg::kStage);
                const uint64_t ad = umb::umma_smem_desc_sw128(st), wd = umb::umma_smem_desc_sw128(st + Cfg::kABytes);
                if (umb::elect_one()) {
#pragma unroll
                    for (int kk = 0; kk < kTcK / 16; ++kk)
                        umb::umma_ss_f16(d, ad + kk * 2, wd + kk * 2, idesc, (k | kk) ? 1u : 0u);
                    umb::umma_commit(empty + s);
                    if (k + 1 == t.k_steps) umb::umma_commit(acc_full + acc);
                }
                ready = __all_sync(0xffffffffu, next);
                s = s2;
                ph = ph2;
            }
        }
    } else if (warp < 2 + Cfg::kStore) {
        constexpr int kPart = kOut / (Cfg::kStore / 4);     // of the columns
        const int q = warp & 3, part = (warp - 2) >> 2;     // the quarter of tensor-memory lanes this warp may read
        float* so = s_out + (warp - 2) * Cfg::kStoreBlock;
        for (uint32_t it = 0; w.step(); ++it) {
            const uint32_t acc = it & 1;
            if (!__all_sync(0xffffffffu, tc_poll(acc_full + acc, (it >> 1) & 1, quit))) break;      // (and the warp is one again)
            umb::tc_fence_after();
            tc_store_tile<kPart, kOut, DUAL, TC, Cfg::kStoreCols>(a, t.vec_c, tmem + acc * BN + part * kPart + ((uint32_t)(q * 32) << 16), so, w.g, w.row_lo + w.m0 + q * 32,
                                          w.rows - w.m0 - q * 32, w.n0 * kOut + part * kPart, [&] { umb::mbar_arrive(acc_empty + acc); });
        }
    } else if (!DENSE) {
        // eight lanes copy a row's 128 bytes of the k step; the image is the one a 128-byte-swizzled TMA box would leave
        constexpr int PW = Cfg::kWarpsPerStage, RS = 4 * PW;                // rows a stage's warps copy side by side
        const int cw = warp - 2 - Cfg::kStore, st = cw / PW, ch = lane & 7, r0 = (cw % PW) * 4 + (lane >> 3);
        int* src = reinterpret_cast<int*>(bars + 32) + cw * kTcRows;        // this warp's list of the tile's source rows
        const __nv_bfloat16* A = (const __nv_bfloat16*)a.A + ch * 8;
        const uint32_t base = smem_u32(smem + st * Cfg::kStage);
        uint32_t uses = 0;
        int unit = 0;                                       // k steps of the tiles before, modulo the ring
        bool ok = true;
        while (ok && w.step()) {
            const int rows = min(kTcRows, w.rows - w.m0);
            __syncwarp();
#pragma unroll
            for (int i = 0; i < kTcRows / 32; ++i) {
                const int r = w.m0 + i * 32 + lane;
                src[i * 32 + lane] = r < w.rows ? (a.row_src ? a.row_src[w.row_lo + r] : w.row_lo + r) : -1;
            }
            __syncwarp();
            const __nv_bfloat16* Ag = A + (t.a_grouped ? (int64_t)w.g * a.a_goff : 0);
            for (int k = (st - unit + kStages) % kStages; k < t.k_steps; k += kStages, ++uses) {
                if (!(ok = __all_sync(0xffffffffu, tc_poll(empty + st, (uses & 1) ^ 1, quit)))) break;
                const int kc = k * kTcK + ch * 8;
                const int bytes = kc < a.K ? 16 : 0;        // behind the last column: zeros (K is a multiple of 8)
                // (rows that are not there keep what the stage held: their sums are not stored)
#pragma unroll 8
                for (int r = r0; r < rows; r += RS)
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(base + r * 128 + ((ch ^ (r & 7)) << 4)),
                                 "l"(Ag + (int64_t)src[r] * a.lda + (bytes ? k * kTcK : 0)), "r"(bytes) : "memory");
                asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
                umb::fence_proxy_async_smem();              // the copies of this thread are complete: show them to the tensor core
                __syncwarp();
                if (lane == 0) umb::mbar_arrive(full + st);
            }
            unit = (unit + t.k_steps) % kStages;
        }
    }
    if (!DENSE && warp >= 2 && warp < 6 && a.rows_total > 0) {             // rows of no group: in front of the first, behind the last
        const int64_t lo = min(a.grp_off[0], a.rows_total), gap = a.grp_off[t.groups] - lo;
        for (int64_t i = (int64_t)blockIdx.x * 4 + warp - 2; i < a.rows_total - gap; i += (int64_t)gridDim.x * 4) {
            const int64_t r = i < lo ? i : i + gap;
            for (int n = lane; n < a.N; n += 32) ((TC*)a.C)[r * a.ldc + n] = from_f32<TC>(0.f);
        }
    }
    __syncthreads();
    tc_settle(quit, t.report);
    if (warp == 1) {
        umb::tc_fence_after();
        umb::tmem_dealloc(tmem, 2 * BN);
    }
}

// ------------------------------------------------------------------------------------------------ host side
static std::atomic<unsigned int*> g_give_up{nullptr};       // 4 bytes for the process, shared by its devices, streams and threads

int give_up_word(unsigned int** word) {
    static std::mutex making;
    unsigned int* w = g_give_up.load(std::memory_order_acquire);
    if (w == nullptr) {
        std::lock_guard<std::mutex> lock(making);
        w = g_give_up.load(std::memory_order_acquire);
        if (w == nullptr) {
            cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;      // (the first call may be inside a capture)
            cudaError_t e = cudaThreadExchangeStreamCaptureMode(&mode);
            if (e != cudaSuccess) return (int)e;
            e = cudaHostAlloc((void**)&w, sizeof *w, cudaHostAllocPortable | cudaHostAllocMapped);
            cudaThreadExchangeStreamCaptureMode(&mode);
            if (e != cudaSuccess) return (int)e;
            *w = 0u;
            g_give_up.store(w, std::memory_order_release);
        }
    }
    *word = w;
    return 0;
}
int give_up_status() {
    const volatile unsigned int* w = g_give_up.load(std::memory_order_acquire);
    return w != nullptr && *w != 0u ? UMB_ERR_TIMEOUT : 0;
}

typedef CUresult (*EncodeTiled)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
static EncodeTiled encode_tiled() {
    static const EncodeTiled fn = [] {
        void* sym = nullptr;
        cudaDriverEntryPointQueryResult q;
        return cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &sym, cudaEnableDefault, &q) == cudaSuccess &&
                       q == cudaDriverEntryPointSuccess ? (EncodeTiled)sym : nullptr;
    }();
    return fn;
}

int encode_map(CUtensorMap* map, const void* base, uint64_t cols, uint64_t rows, uint64_t groups, uint64_t ld, uint64_t gs,
                      uint32_t box_rows) {
    const EncodeTiled enc = encode_tiled();
    if (enc == nullptr) return UMB_ERR_DRIVER;
    const cuuint64_t dims[3] = {cols, rows, groups}, strides[2] = {ld * 2, (groups > 1 ? gs : ld * rows) * 2};
    const cuuint32_t box[3] = {64, box_rows, 1}, one[3] = {1, 1, 1};
    return enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(base), dims, strides, box, one, CU_TENSOR_MAP_INTERLEAVE_NONE,
               CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS
               ? 0 : UMB_ERR_DRIVER;
}

template <int BN, bool DUAL, bool DENSE, typename TC>
static int launch_tc(const GemmArgs& a, TcArgs t, const CUtensorMap& ma, int sms, cudaStream_t st) {
    using Cfg = TcCfg<BN, DUAL>;
    t.n_tiles = (a.N + Cfg::kOut - 1) / Cfg::kOut;
    t.k_steps = (a.K + kTcK - 1) / kTcK;
    const int gw = a.w_gstride != 0 ? t.groups : 1;
    t.w_grouped = gw > 1;
    CUtensorMap mw;
    const int rc = encode_map(&mw, a.W, a.K, (uint64_t)a.N * (DUAL ? 2 : 1), gw, a.ldw, a.w_gstride, Cfg::kOut);
    if (rc != 0) return rc;
    auto kernel = gemm_tc_kernel<BN, DUAL, DENSE, TC>;
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::kSmem);
    if (e != cudaSuccess) return (int)e;
    const int64_t tiles = (int64_t)t.groups * t.m_tiles * t.n_tiles;            // (sorted by expert: at most)
    return chain_launch(kernel, (int)(tiles < sms ? tiles : sms), Cfg::threads(DENSE), Cfg::kSmem, st, ma, mw, a, t);
}

template <int BN>
static int launch_tc_any(const GemmArgs& a, TcArgs t, bool dual, bool c_f32, int sms, cudaStream_t st) {
    const int ga = a.a_goff != 0 ? t.groups : 1;
    const bool dense = a.grp_off == nullptr && a.row_src == nullptr;
    t.a_grouped = ga > 1;
    CUtensorMap ma{};
    if (dense) {
        const int rc = encode_map(&ma, a.A, a.K, a.M, ga, a.lda, a.a_goff, kTcRows);
        if (rc != 0) return rc;
    }
#define UMBS_TC(D, S) (c_f32 ? launch_tc<BN, D, S, float>(a, t, ma, sms, st) : launch_tc<BN, D, S, __nv_bfloat16>(a, t, ma, sms, st))
    if (dual) return dense ? UMBS_TC(true, true) : UMBS_TC(true, false);
    return dense ? UMBS_TC(false, true) : UMBS_TC(false, false);
#undef UMBS_TC
}

// The tile width with the shortest longest walk.  Dense rows, in ns: what a launch, a tile's first operands and its last results take,
// and a k step of a round of tiles (measured, loaded chip; pairs of SMs: seq_gemm_pair.cu).  us, single blocks / pairs: 803 rows, K =
// 1024, to 1024 / 3088 columns 8.6 / 12.1, 15.2 / 13.3; 1500, K = 2048, to 6144 34.9 / 31.0; 4096 90.0 / 80.1; 4096, K = 1024, to 4096
// 41.8 / 34.1.
// Rows sorted by expert (how they fall is only known on the device; spread evenly is the guess): rounds of tiles times what 16 of k
// cost, the tensor core's 128 clocks for 256 columns and more than half, a quarter of that for 128 and 64: 72 and 52 (the activation
// tile is fetched and read from shared memory for fewer products).
int tc_tile_columns(int M, int N, int K, int groups, bool dual, bool by_group, bool gathered, int sms) {
    const bool dense = !by_group && !gathered;
    const int64_t m = by_group ? (int64_t)groups * ((M + groups * kTcRows - 1) / (groups * kTcRows)) : (int64_t)groups * ((M + kTcRows - 1) / kTcRows);
    const int64_t steps = dense ? (K + kTcK - 1) / kTcK : 1;
    auto cost = [&](int bn, int step, int once) {
        const int out = dual ? bn / 2 : bn;
        return (m * ((N + out - 1) / out) + sms - 1) / sms * steps * step + (dense ? once : 0);
    };
    const int64_t c256 = cost(256, dense ? 410 : 128, 8300), c128 = cost(128, dense ? 275 : 72, 6000), c64 = cost(64, dense ? 250 : 52, 4300);
    if (dense && M > kTcRows) {
        const int out = dual ? 128 : 256;
        const int64_t tiles = (int64_t)groups * ((M + 255) / 256) * ((N + out - 1) / out), pair = (tiles + sms / 2 - 1) / (sms / 2) * steps * 370 + 6800;
        if (pair < c256 && pair < c128 && pair < c64) return UMBS_GEMM_PAIRS;
    }
    if (c256 <= c128 && c256 <= c64) return 256;
    return c128 <= c64 ? 128 : 64;
}

int launch_gemm_tc(const GemmArgs& a, int groups, bool dual, bool c_f32, cudaStream_t st) {
    int dev = 0, sms = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return (int)e;
    TcArgs t{};
    int rc = give_up_word(&t.report);
    if (rc == 0) rc = give_up_status();
    if (rc != 0) return rc;
    t.groups = groups;
    t.m_tiles = (a.M + kTcRows - 1) / kTcRows;
    const int es = c_f32 ? 4 : 2;
    t.vec_c = (uintptr_t)a.C % (4 * es) == 0 && a.ldc % 4 == 0 && a.c_goff % 4 == 0;
    switch (tc_tile_columns(a.M, a.N, a.K, groups, dual, a.grp_off != nullptr, a.row_src != nullptr, sms)) {
        case UMBS_GEMM_PAIRS: return launch_gemm_pair(a, t, dual, c_f32, sms, st);
        case 256: return launch_tc_any<256>(a, t, dual, c_f32, sms, st);
        case 128: return launch_tc_any<128>(a, t, dual, c_f32, sms, st);
        default: return launch_tc_any<64>(a, t, dual, c_f32, sms, st);
    }
}

}  // namespace umbs

extern "C" unsigned int umbs_give_ups_seen(void) { return umbs::give_up_status() != 0; }
extern "C" unsigned int umbs_kernel_timeouts(void) { return umbs::tc_timeouts() + umbs::attention_tc_timeouts() + umbs::split_timeouts() + umbs::pair_timeouts() + umbs::chunk_tc_timeouts(); }
