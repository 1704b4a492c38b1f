// AWQ INT4 products of 129 to 512 token rows by pairs of SMs (tcgen05 cta_group::2), for prompts and wide trees.
//
// Weights are the A operand as in gemm.cu, but of two tiles at once: each block of a pair dequantises the records of its own 128
// output features into its own tensor memory, holds half of the token rows of a slab of 128 k in shared memory, and the tensor
// cores of both multiply 256 features with up to 256 rows (M = 256, N = 192 or 256).  A record is dequantised once for up to 256 rows and
// a slab's bytes cross into an SM once for 256 features.
//
// Warp roles of a block (480 threads, one block per SM):
//   warp 0        weight records, one bulk copy each (ahead of griddepcontrol.wait: weights depend on nothing in the stream)
//   warp 1        its half of the x slabs, counted by the first block's barrier
//   warp 2        (first block) issues the products of both
//   warps 3-10    two dequant groups: shared memory -> registers -> tensor memory, as in gemm.cu
//   warps 11-14   a third group: all three finish tiles, 16 token columns each in turn
// The work is cut into equal contiguous ranges of units (pair of tiles, block of rows, 128 k), one range per pair.  Of a tile that ranges
// share, a pair that goes on to other tiles publishes its sums in the workspace; those that end with it divide the columns among them, 16 at
// a time in turn: each publishes the others' columns, keeps its own in tensor memory and adds the parts to them in ascending order of the ranges
// (deterministic).  A published fp32 word is its own flag (0 = not written yet), and no pair waits for another while it has products to do.
// (All parts through the workspace, added up by all pairs: 4 x 128 KB a block written, read and cleared at the same time, 18 us of 107 for
// 4096 -> 28672 and 500 rows.)
//
// Bound: a unit takes 610 to 650 ns, its products 540 at the measured cuBLAS rate; the next tile's products wait for the columns of the one
// before (5 us where it is published, 10 where it is finished: the accumulator fills half of tensor memory, so there is one), and the end of
// a range is 12 us of 100.  us, four passes of 125 rows through gemm.cu's kernel / one of 500 here: a layer of width 4096 and its head, weights from memory, 695 / 456, of width
// 8192 1363 / 1129 (its 28672 k in passes); width 4096, 1000 rows 1244 / 757, 300 540 / 374, 129 376 / 304.  Up to 128 rows, one pass on both sides, this gains nothing (gemm.cu does them).  Of no effect: fewer records, fewer or no x
// copies, no arithmetic in the dequantisation (2 to 8 % each), deeper record rings.
#include "gemm_core.cuh"
#include "group_gate.h"

namespace umb {
namespace {

constexpr int kWideThreads = 96 + 3 * 128;
constexpr int kWideW = 8;                                   // records held
constexpr int kWideRecord = 8576;                           // a record in shared memory, padded to 128 bytes
constexpr int kWideExch = 16 * 128 * 2;                     // a group's rows in epilogue_chunk (without rows of cos and sin)
constexpr int kWideSlots = 2;                               // parts of tiles that a block publishes: of the tile it begins within, of its last
template <int NPAD> struct WideCfg {
    static constexpr int kRows = NPAD / 2;                  // rows of a slab that a block holds
    static constexpr int kXBytes = kRows * 256;             // [2 pieces of 64 k][rows][128 B]
    static constexpr int kX = (512 - NPAD) / 128 * 2;       // x slabs, and parts of the A operand (64 columns each, behind the accumulator)
    static constexpr int kSmem = 1024 + kX * kXBytes + kWideW * kWideRecord + 3 * kWideExch;
};

__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_sync() { asm volatile("barrier.cluster.arrive.aligned;\n\tbarrier.cluster.wait.aligned;" ::: "memory"); }
__device__ __forceinline__ uint32_t first_block(const void* p) {            // the first block's copy of a shared variable
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(r) : "r"(smem_u32(p)));
    return r;
}
__device__ __forceinline__ void arrive_at(uint32_t bar) {
    asm volatile("mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tma_3d_pair(void* dst, const CUtensorMap* map, int c0, int c1, int c2, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
                 ::"r"(smem_u32(dst)), "l"(map), "r"(c0), "r"(c1), "r"(c2), "r"(bar) : "memory");
}
__device__ __forceinline__ void umma_pair_ts(uint32_t d, uint32_t a, uint64_t bd, uint32_t idesc, uint32_t accumulate) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
                 ::"r"(d), "r"(a), "l"(bd), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void commit_pair(uint64_t* bar) {                // the same barrier of both blocks
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
                 ::"r"(smem_u32(bar)), "h"((uint16_t)3) : "memory");
}

// Every wait is bounded (seconds): a block that gives up raises its flag and all of its roles leave their loops.
__device__ __forceinline__ bool give_up(volatile int* quit) {
    *quit = 1;
    return false;
}
// PAIR: a barrier that the other block's threads, or products of both, arrive at.  What such a barrier hands over is in tensor memory, or the products' reads of
// shared memory are over: the fences of tcgen05 on both sides order that, and the barrier itself is relaxed, but in cluster scope.  (Arrivals that release
// in cluster scope: a prompt of 500 rows 470 -> 500 us; every look acquiring in it: 1.5 times the whole.)
#define UMB_TEST_WAIT(PAIR) "mbarrier.test_wait.parity" PAIR ".shared::cta.b64 p, [%1], %2;\n\t"
template <bool PAIR>
__device__ __forceinline__ bool test_bar(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    if constexpr (PAIR)
        asm volatile("{\n\t.reg .pred p;\n\t" UMB_TEST_WAIT(".relaxed.cluster") "selp.u32 %0, 1, 0, p;\n\t}" : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity) : "memory");
    else
        asm volatile("{\n\t.reg .pred p;\n\t" UMB_TEST_WAIT("") "selp.u32 %0, 1, 0, p;\n\t}" : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity) : "memory");
    return ok != 0;
}
template <bool PAIR>
__device__ __forceinline__ bool poll_bar(uint64_t* bar, uint32_t parity, volatile int* quit) {
    bool ok = false;
    for (int i = 0; i < (1 << 24); ++i) {
        if ((ok = test_bar<PAIR>(bar, parity))) break;
        __nanosleep(20);
        if ((i & 255) == 255 && *quit) break;
    }
    return __all_sync(0xffffffffu, ok) || give_up(quit);
}
__device__ __forceinline__ bool wait_bar(uint64_t* bar, uint32_t parity, volatile int* quit) { return poll_bar<false>(bar, parity, quit); }
__device__ __forceinline__ bool wait_pair(uint64_t* bar, uint32_t parity, volatile int* quit) { return poll_bar<true>(bar, parity, quit); }
// without a pause, for the warp that issues the products (one statement: as C++ the loop's exits cost 100 clocks a wait)
#define UMB_SPIN(PAIR)                                                                                         \
    uint32_t ok;                                                                                               \
    asm volatile(                                                                                              \
        "{\n\t.reg .pred p, q;\n\t.reg .u32 n;\n\tmov.u32 n, 0;\n\t"                                           \
        "AGAIN_%=:\n\t" UMB_TEST_WAIT(PAIR)                                                                    \
        "@p bra DONE_%=;\n\t"                                                                                  \
        "add.u32 n, n, 1;\n\tsetp.lt.u32 q, n, 67108864;\n\t@q bra AGAIN_%=;\n\t"                              \
        "DONE_%=:\n\tselp.u32 %0, 1, 0, p;\n\t}"                                                               \
        : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity) : "memory");                                              \
    return __all_sync(0xffffffffu, ok) || give_up(quit);
__device__ __forceinline__ bool spin_bar(uint64_t* bar, uint32_t parity, volatile int* quit) { UMB_SPIN("") }
__device__ __forceinline__ bool spin_pair(uint64_t* bar, uint32_t parity, volatile int* quit) { UMB_SPIN(".relaxed.cluster") }
#undef UMB_SPIN
#undef UMB_TEST_WAIT
// The four warps of a group go on together or not at all (GroupGate): what follows holds barriers of theirs.
__device__ __forceinline__ bool group_all(bool ok, int bar) {
    int all = ok;
    asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.s32 p, %0, 0;\n\tbarrier.cta.red.and.pred q, %1, 128, p;\n\tselp.s32 %0, 1, 0, q;\n\t}"
                 : "+r"(all) : "r"(bar) : "memory");
    return all != 0;
}
__device__ __forceinline__ uint4 ld_words(const uint32_t* p) {
    uint4 v;
    asm volatile("ld.relaxed.gpu.global.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory");
    return v;
}

struct WideRows { int shift, rows; };                       // 2^shift blocks of token rows, rows of a block (a multiple of 16)

template <int NPAD>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kWideThreads, 1)
awq_wide_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ GemmParams p, const WideRows rb, volatile unsigned int* report) {
    using Cfg = WideCfg<NPAD>;
    constexpr int kX = Cfg::kX, kACol = NPAD;               // first column of the A operand's parts
    extern __shared__ unsigned char smem_raw[];
    __shared__ uint64_t bars[2 * kWideW + 3 * kX + 3];
    __shared__ uint32_t s_tmem;
    __shared__ int s_quit;
    unsigned char* s_x = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    unsigned char* s_w = s_x + kX * Cfg::kXBytes;
    __half* s_exch = reinterpret_cast<__half*>(s_w + kWideW * kWideRecord);
    uint64_t *full_w = bars, *empty_w = full_w + kWideW,    // this block's records: landed, in registers
             *full_x = empty_w + kWideW,                    // (first block) both halves of a slab
             *full_a = full_x + kX,                         // (first block) both blocks' parts of the A operand
             *done = full_a + kX,                           // the unit's products are over: its slab and its part of A are free
             *acc_full = done + kX, *acc_empty = acc_full + 1,           // a segment's sums; (first block) they have been read
             *last_full = acc_full + 2;                     // the last segment's
    volatile int* quit = &s_quit;
    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
    const int rank = (int)cluster_rank();
    if (threadIdx.x == 0) {
        tma_prefetch_desc(&map_x);
        for (int i = 0; i < kWideW; ++i) {
            mbar_init(full_w + i, 1);
            mbar_init(empty_w + i, 4);
        }
        for (int i = 0; i < kX; ++i) {
            mbar_init(full_x + i, 1);
            mbar_init(full_a + i, 8);
            mbar_init(done + i, 1);
        }
        mbar_init(acc_full, 1);
        mbar_init(acc_empty, 24);
        mbar_init(last_full, 1);
        s_quit = 0;
        fence_barrier_init();
    }
    if (warp == 2) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(&s_tmem)) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;");
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync();                                         // both blocks' barriers are there
    tc_fence_after();
    pdl_launch_dependents();
    const uint32_t tmem = s_tmem;

    // the pair's units; a tile is (pair of tiles, block of rows), blocks fastest
    const int G = p.units_per_tile, me = (int)(blockIdx.x >> 1);
    const long long U = (long long)((p.tiles + 1) / 2) * (1 << rb.shift) * G, P = gridDim.x >> 1;
    const long long u_begin = sk_begin(me, U, P), u_end = sk_begin(me + 1, U, P);
    const int n_units = (int)(u_end - u_begin), t_first = (int)(u_begin / G), g_first = (int)(u_begin - (long long)t_first * G);

    if (warp == 0) {
        // ------------------------------------------------------------------------------------ weight records
        // (a second tile that does not exist: the last one's records, and nothing is stored)
        auto record = [&](int t, int g) { return p.packed + ((size_t)min(2 * (t >> rb.shift) + rank, p.tiles - 1) * G + g) * kRecordStride; };
        const uint64_t pol = l2_policy_evict_first();
        int t = t_first, g = g_first;
        const unsigned char* src = record(t, g);
        for (int i = 0; i < n_units; ++i) {
            const int s = i % kWideW;
            if (i >= kWideW && !wait_bar(empty_w + s, ((i / kWideW) - 1) & 1, quit)) break;
            if (elect_one()) {
                mbar_arrive_expect_tx(full_w + s, kRecordBytes);
                tma_bulk_g2s(s_w + s * kWideRecord, src, kRecordBytes, full_w + s, pol);
            }
            __syncwarp();
            src += kRecordStride;
            if (++g == G) {
                g = 0;
                src = record(++t, 0);
            }
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------------------------------ x slabs
        pdl_wait();
        int g = g_first, row = (t_first & ((1 << rb.shift) - 1)) * rb.rows;
        for (int i = 0; i < n_units; ++i) {
            const int s = i % kX;
            if (i >= kX && !wait_pair(done + s, ((i / kX) - 1) & 1, quit)) break;
            const uint32_t bar = first_block(full_x + s);
            if (elect_one()) {
                if (rank == 0) mbar_arrive_expect_tx(full_x + s, 2 * Cfg::kXBytes);
                tma_3d_pair(s_x + s * Cfg::kXBytes, &map_x, 0, row + rank * Cfg::kRows, g * 2, bar);
            }
            __syncwarp();
            if (++g == G) {
                g = 0;
                row += rb.rows;
                if (row >= (1 << rb.shift) * rb.rows) row = 0;
            }
        }
    } else if (warp == 2) {
        // ------------------------------------------------------------------------------------ products
        if (rank == 0) {
            constexpr uint32_t idesc = umma_idesc_f16(256, NPAD);
            int in_tile = g_first, seg = 0, u = 0;
            bool ok = true;
            while (ok && u < n_units) {
                const int end = u + min(n_units - u, G - in_tile);
                if (seg > 0 && !(ok = spin_pair(acc_empty, (seg - 1) & 1, quit))) break;
                for (const int first = u; u < end; ++u) {
                    const int s = u % kX, ph = (u / kX) & 1;
                    if (!(ok = spin_bar(full_x + s, ph, quit)) || !(ok = spin_pair(full_a + s, ph, quit))) break;
                    tc_fence_after();
                    const uint64_t bd = umma_smem_desc_sw128(smem_u32(s_x + s * Cfg::kXBytes));
                    const uint32_t a = tmem + kACol + s * 64;
                    if (elect_one()) {
#pragma unroll
                        for (int kk = 0; kk < 8; ++kk)
                            umma_pair_ts(tmem, a + kk * 8, bd + (uint64_t)(((kk >> 2) * (Cfg::kRows * 128) + (kk & 3) * 32) >> 4), idesc,
                                         (u > first || kk > 0) ? 1u : 0u);
                        commit_pair(done + s);
                        if (u + 1 == end) commit_pair(end == n_units ? last_full : acc_full);
                    }
                    __syncwarp();
                }
                in_tile = 0;
                ++seg;
            }
        }
    } else {
        const int grp = (warp - 3) >> 2;                    // 0 and 1 dequantise, all three finish tiles
        const int q = warp & 3, fl = q * 32 + lane;         // quarter of tensor memory, feature of the tile
        const uint32_t quarter = tmem + ((uint32_t)(q * 32) << 16);
        __half* exch = s_exch + grp * (kWideExch / 2);
        GroupGate gate;
        auto together = [&](bool ok) { return gate.pass(ok, [&](bool mine) { return group_all(mine, 1 + grp); }); };
        // words of a part: [4 token columns][feature][4]; which: 0 of the tile that the range begins within, 1 of a tile that it begins
        auto slot = [&](int c, int which) {
            return reinterpret_cast<uint32_t*>(p.slots) + ((size_t)(c * 2 + rank) * kWideSlots + which) * ((size_t)NPAD * kTileN) + fl * 4;
        };
        auto rows_of = [&](int t) { return min(rb.rows, p.M - (t & ((1 << rb.shift) - 1)) * rb.rows); };
        auto publish = [&](uint32_t* part, int j, int rows) {                       // columns 16 j ..
            uint32_t rr[16];
            UMB_TMEM_LD_X16(quarter + j * 16, rr);
            tc_wait_ld();
#pragma unroll
            for (int e = 0; e < 16; ++e) rr[e] = rr[e] ? rr[e] : 0x80000000u;       // (+0 leaves as -0, which adds the same)
#pragma unroll
            for (int e = 0; e < 4; ++e)
                if (j * 16 + e * 4 < rows) *reinterpret_cast<uint4*>(part + (j * 16 + e * 4) * kTileN) = make_uint4(rr[4 * e], rr[4 * e + 1], rr[4 * e + 2], rr[4 * e + 3]);
        };
        auto to_rows = [&](int t, int j, const float (&v)[16]) {
            epilogue_chunk(p, 2 * (t >> rb.shift) + rank, fl, (t & ((1 << rb.shift) - 1)) * rb.rows + j * 16, v, exch, 1 + grp);
        };
        // A tile that is not the range's last, by all three groups: finished when it is whole, else published (it is the first, and its
        // other parts are not this pair's to add).
        auto leave_tile = [&](int t) -> bool {
            if (!together(wait_pair(acc_full, (t - t_first) & 1, quit))) return false;
            tc_fence_after();
            const int rows = rows_of(t);
            const bool whole = t > t_first || g_first == 0;
            uint32_t* part = slot(me, 0);
            if (!whole)
                for (int j = grp; j * 16 < rows; j += 3) publish(part, j, rows);
            auto free_columns = [&] {
                tc_fence_before();
                __syncwarp();
                if (lane == 0) arrive_at(first_block(acc_empty));
            };
            for (int j = grp; whole && j * 16 < rows; j += 3) {
                float v[16];
                uint32_t rr[16];
                UMB_TMEM_LD_X16(quarter + j * 16, rr);
                tc_wait_ld();
                if ((j + 3) * 16 >= rows) free_columns();
#pragma unroll
                for (int e = 0; e < 16; ++e) v[e] = __uint_as_float(rr[e]);
                to_rows(t, j, v);
            }
            if (!whole || grp * 16 >= rows) free_columns();
            return true;
        };
        const int t_last = n_units > 0 ? (int)((u_end - 1) / G) : t_first;
        bool ok = true;
        int t = t_first;                                    // a tile whose sums are not read yet
        if (grp < 2) {
            // -------------------------------------------------------------------------------- dequantise units grp, grp + 2, ...
            int t_end = G - g_first;                        // the unit behind tile t
            for (int i = grp; ok && i < n_units; i += 2) {
                // what is ahead needs the products of units behind t_end, which wait for the accumulators
                if (t < t_last && i - kX >= t_end) {
                    pdl_wait();                             // (the workspace belongs to the kernels in front)
                    for (; ok && t < t_last && i - kX >= t_end; ++t, t_end += G) ok = leave_tile(t);
                    if (!ok) break;
                }
                const int ws = i % kWideW, as = i % kX;
                if (!(ok = wait_bar(full_w + ws, (i / kWideW) & 1, quit))) break;
                const uint32_t rec = smem_u32(s_w + ws * kWideRecord);
                uint4 w4[4];
#pragma unroll
                for (int c = 0; c < 4; ++c) w4[c] = lds128(rec + (c * kTileN + fl) * 16);
                const uint32_t sbits = lds16(rec + kRecScaleOff + fl * 2), z = (lds32(rec + kRecZeroOff + (fl >> 3) * 4) >> (4 * (fl & 7))) & 0xFu;
                __syncwarp();
                if (lane == 0) mbar_arrive(empty_w + ws);
                if (i >= kX && !(ok = wait_pair(done + as, ((i / kX) - 1) & 1, quit))) break;
                tc_fence_after();
                const __half2 ce = as_h2((0x6400u | z) * 0x10001u), neg_co = as_h2((0xD400u | (z << 4)) * 0x10001u), s2 = as_h2(sbits * 0x10001u);
                const uint32_t to = quarter + kACol + as * 64;
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    const uint32_t words[4] = {w4[c].x, w4[c].y, w4[c].z, w4[c].w};
                    uint32_t a[16];
#pragma unroll
                    for (int w = 0; w < 4; ++w) dequant_word(words[w], 0x64006400u, ce, neg_co, s2, &a[w * 4]);
                    UMB_TMEM_ST_X16(to + c * 16, a);
                }
                tc_wait_st();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) arrive_at(first_block(full_a + as));
            }
        }
        pdl_wait();                                         // residual, workspace and y belong to the kernels in front
        for (; ok && t < t_last; ++t) ok = leave_tile(t);
        // ------------------------------------------------------------------------------------ the range's last tile
        ok = together(ok && n_units > 0 && wait_pair(last_full, 0, quit));
        if (ok) {
            tc_fence_after();
            const int rows = rows_of(t);                    // (t is t_last)
            const long long u0 = (long long)t * G;
            const int c0 = sk_owner(u0, U, P), c1 = sk_owner(u0 + G - 1, U, P);
            const int ends = sk_begin(c1 + 1, U, P) > u0 + G ? c1 - c0 : c1 - c0 + 1;            // pairs c0 .. c0 + ends - 1 end with this tile
            uint32_t* part = slot(me, me == c0 ? 1 : 0);
            if (ends > 1)
                for (int j = grp; j * 16 < rows; j += 3)
                    if (j % ends != me - c0) publish(part, j, rows);
            // this group's turns; parts in ascending order, the words of the next on their way while one is added
            uint4 w[4];
            auto load = [&](int c, int j) {
                const uint32_t* src = slot(c, c == c0 ? 1 : 0) + j * (16 * kTileN);
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    w[e] = make_uint4(0x80000000u, 0x80000000u, 0x80000000u, 0x80000000u);
                    if (j * 16 + e * 4 < rows) w[e] = ld_words(src + e * (4 * kTileN));
                }
            };
            const int first = c0 != me ? c0 : c0 + 1;       // (beyond c1: there is no other part)
            for (int j = me - c0 + ends * grp; ok && j * 16 < rows; j += 3 * ends) {
                if (first <= c1) load(first, j);
                uint32_t own[16];
                UMB_TMEM_LD_X16(quarter + j * 16, own);
                tc_wait_ld();
                float v[16];
#pragma unroll
                for (int e = 0; e < 16; ++e) v[e] = me == c0 ? __uint_as_float(own[e]) : 0.f;
                for (int c = first; ok && c <= c1; ++c) {
                    if (c == me) {
#pragma unroll
                        for (int e = 0; e < 16; ++e) v[e] += __uint_as_float(own[e]);
                        continue;
                    }
                    for (int n = 0;; ++n) {
                        uint32_t least = 0xffffffffu;
#pragma unroll
                        for (int e = 0; e < 4; ++e) least = min(least, min(min(w[e].x, w[e].y), min(w[e].z, w[e].w)));
                        if (__all_sync(0xffffffffu, least != 0u)) break;
                        if (__any_sync(0xffffffffu, n == (1 << 22) || *quit)) {
                            ok = give_up(quit);
                            break;
                        }
                        load(c, j);
                    }
                    uint32_t* src = slot(c, c == c0 ? 1 : 0) + j * (16 * kTileN);
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        v[4 * e] += __uint_as_float(w[e].x);
                        v[4 * e + 1] += __uint_as_float(w[e].y);
                        v[4 * e + 2] += __uint_as_float(w[e].z);
                        v[4 * e + 3] += __uint_as_float(w[e].w);
                        if (j * 16 + e * 4 < rows) *reinterpret_cast<uint4*>(src + e * (4 * kTileN)) = make_uint4(0u, 0u, 0u, 0u);      // (handed on clean)
                    }
                    const int next = c + 1 == me ? c + 2 : c + 1;
                    if (next <= c1) load(next, j);
                }
                if (!(ok = together(ok))) break;
                to_rows(t, j, v);
            }
        }
    }
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    if (*quit) {                                            // copies and products in flight end before their memory goes
        if (threadIdx.x == 0) {
            *report = 1u;
            __threadfence_system();
        }
        for (int i = 0; i < 1000; ++i) __nanosleep(1000);
    }
    __syncthreads();
    cluster_sync();                                         // neither block's memory goes while the other's products or copies use it
    if (warp == 2) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, 512;" ::"r"(tmem));
    }
}

template <int NPAD>
int launch_wide(const void* x, int64_t ldx, GemmParams p, WideRows rb, cudaStream_t st) {
    p.rope_vec_ok = 0;                                      // (kWideExch)
    unsigned int* report = nullptr;
    int rc = give_up_word(&report);
    if (rc != UMB_OK) return rc;
    CUtensorMap map;
    rc = make_tmap_x3d(&map, x, (uint64_t)p.M, (uint64_t)p.K, (uint64_t)ldx, WideCfg<NPAD>::kRows);
    if (rc != UMB_OK) return rc;
    const long long units = (long long)((p.tiles + 1) / 2) * (1 << rb.shift) * p.units_per_tile;
    const int pairs = (int)(units < sm_count() / 2 ? units : sm_count() / 2);
    UMB_CUDA(cudaFuncSetAttribute(awq_wide_kernel<NPAD>, cudaFuncAttributeMaxDynamicSharedMemorySize, WideCfg<NPAD>::kSmem));
    UMB_LAUNCH_PDL(awq_wide_kernel<NPAD>, dim3(2 * pairs), dim3(kWideThreads), (size_t)WideCfg<NPAD>::kSmem, st, map, p, rb, report);
    count_launches(1);
    return UMB_OK;
}

// blocks of equal height, as few as the accumulator's 256 columns allow
WideRows wide_rows(int M) {
    const int shift = M > 256 ? 1 : 0;
    return {shift, (((M + shift) >> shift) + 15) / 16 * 16};
}
int wide_columns(int rows) { return rows <= 192 ? 192 : 256; }

}  // namespace

size_t awq_wide_ws_bytes(int M, int N_total) {
    const size_t tiles = (size_t)(N_total + kTileN - 1) / kTileN;
    return ((tiles * 4 + 255) & ~(size_t)255) + (size_t)2 * (sm_count() / 2) * kWideSlots * wide_columns(wide_rows(M).rows) * kTileN * sizeof(float);
}

int launch_awq_wide(const void* x, int64_t ldx, const GemmParams& p, cudaStream_t st) {
    const WideRows rb = wide_rows(p.M);
    return wide_columns(rb.rows) == 192 ? launch_wide<192>(x, ldx, p, rb, st) : launch_wide<256>(x, ldx, p, rb, st);
}

}  // namespace umb
