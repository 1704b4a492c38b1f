// Attention of a step with several tokens per sequence on the 5th-generation tensor cores, bf16 storage: the tile kernels of
// seq_cached_attn.cu and seq_window_attn.cu for the sizes and addresses it takes.
//
// A block = 128 consecutive query rows of one (sequence, head) = the 128 lanes of tensor memory; two blocks share an
// SM.  Tiles of 64 keys:
//   warps 9-10 bring key and value rows into the 128-byte-swizzled images the tensor core reads, ahead of their use: with TMA
//              where the 64 rows are neighbours in the step or in the ring, else (the tile between the two, pooled blocks) with
//              16-byte cp.async, each row from where it lives (step, ring, block table), zeros where there is none;
//   warp 8     one thread issues S = Q K^T of the next tile, then O += P V of this one, accumulators in tensor memory;
//   warps 0-7  two threads per row, 32 keys each: scores to weights in fp32 in the base-2 domain, an online reference that only moves
//              when a score of either passes it by 2^8 (then O is rescaled, half of its columns each), the row's sum.
// Weights stay 32-bit: an fp32 weight is the sum of three bf16 numbers (8 + 8 + 8 significant bits, cut off one after the
// other, so exactly), and P V is three products against the same values.  Products of bf16 operands are exact in the tensor
// core and its sums are fp32.
//
// Tensor memory, 256 columns: two score tiles 0-63 and 64-127, in each the first and second parts of its weights over the scores of the
// same thread (0-15 and 16-31, 32-47 and 48-63), output 128-255; third parts in shared memory.  So the next tile's scores are there when a
// tile's weights are done.  (Tiles of 32 keys, a thread per row, all parts in tensor memory: a product of 128 x 32 x 16
// takes the tensor core 48 clocks like one of 128 x 64 x 16, and the thread's chain 1450 of a tile's 2400.  64 keys with all parts in tensor memory
// and one score tile, so that scores, weights and output products take turns: 4500 per tile, with one thread per row 5800.)
//
// Bound: two blocks take 2200 to 2400 ns a tile each (one alone 1650): a row's weights behind the scores and in front of the products (560 instructions a
// warp and tile, issue slots 56 % taken, tensor pipe 39 % active), and blocks that fill the SMs 1.7 times.  us, 32 keys a tile / this: 4096 tokens, 16 heads of 128 over 4 key/value heads,
// window 1024, pooled blocks 115 / 101; two prompts of 2000 tokens, 16 heads of 128 + 64 shared, a gate per column 156 / 106 (blocks that see most keys first,
// over all heads: 40 of it); 106 tokens behind 700, heads of 96, 49 / 32.  A short prompt's block runs every instruction once, and what it waits for is the next
// ones (2500 clocks for the first tile's weights): eight prompts of 20 tokens, 16 heads of 64 over 2, 6.9 / 7.3; three of 77 7.5 / 7.9; 300 tokens, heads of 128, 15.5 / 13.7 (508 calls:
// 1.37 times as fast in the median, 15 of them 3 to 8 % slower).
#include <algorithm>

#include "seq_attn.h"
#include "seq_tc.cuh"

namespace umbs {

constexpr int kTaQ = 128, kTaK = 64;
constexpr int kTaThreads = 352;                             // 8 warps of weights, 1 of products, 2 of copies
constexpr int kTaHeld = 2;                                  // key and value tiles held, at most
constexpr float kTaLazy = 8.f;                              // how far (in powers of two) a score may pass the reference

// 64-wide pieces of a query row, 16-wide k steps, 64-wide pieces of a value row; key tiles and value tiles held; rows of the ring's map; give_up_word()
struct TaDims { int q_atoms, k_steps, v_atoms, k_held, v_held, tma; int64_t ring_rows; unsigned int* report; };

__device__ __forceinline__ float ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ void cp16(uint32_t dst, const void* src, int bytes) {      // fewer than 16 bytes: zeros
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
// the top halves of two words: two bf16 numbers, cut off
__device__ __forceinline__ uint32_t hi_pair(float a, float b) { return __byte_perm(__float_as_uint(a), __float_as_uint(b), 0x7632); }
__device__ __forceinline__ float minus_cut(float a) { return __uint_as_float((__float_as_uint(a) & 0xffff0000u) ^ 0x80000000u); }

// The two warps of a row's threads.
__device__ __forceinline__ void pair_sync(int bar) { asm volatile("bar.sync %0, 64;" ::"r"(bar) : "memory"); }
__device__ __forceinline__ bool pair_all(int bar, bool ok) {                // they go on together or not at all
    int all = ok;
    asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.s32 p, %0, 0;\n\tbarrier.cta.red.and.pred q, %1, 64, p;\n\tselp.s32 %0, 1, 0, q;\n\t}"
                 : "+r"(all) : "r"(bar) : "memory");
    return all != 0;
}
// The key tiles of a block: pooled blocks first, then tokens.
struct KeyTiles {
    int n_pool, tiles_pool, j_lo, p_hi, n;
    __device__ KeyTiles(const CachedAttnArgs& a, int window, int pos0, int q0, int len) {
        const int p_lo = pos0 + q0;
        p_hi = pos0 + min(len, q0 + kTaQ) - 1;
        n_pool = pooled_visible(p_hi, window, a.pool);
        tiles_pool = (n_pool + kTaK - 1) / kTaK;
        j_lo = max(max(0, p_lo - window + 1), a.chunk > 0 ? p_lo / a.chunk * a.chunk : 0);
        n = tiles_pool + (p_hi - j_lo) / kTaK + 1;
    }
    __device__ bool pooled(int i) const { return i < tiles_pool; }
    __device__ int base(int i) const { return i < tiles_pool ? i * kTaK : j_lo + (i - tiles_pool) * kTaK; }
    __device__ int last(int i) const { return i < tiles_pool ? n_pool - 1 : p_hi; }
};

// Row r of (sequence s, virtual head vh) in plain fp32, by a whole warp: the keys it sees, in order, as the kernel below ends.
template <int MODE, bool STEP>
__device__ __noinline__ void plain_row(const CachedAttnArgs& a, const StepKeys& x, const Batch& b, int s, int vh, int r) {
    const int lane = threadIdx.x & 31, start = b.seq_start[s], pos0 = STEP ? 0 : b.seq_pos0[s], slot = STEP ? 0 : b.seq_slot[s], rp = pos0 + r;
    const int window = a.window > 0 ? a.window : (1 << 30);
    const int64_t t = start + r;
    VHead v;
    if (STEP) { v.h = vh; v.qoff = vh * a.dim; }
    else v = virtual_head(a, vh);
    PlainRow p;
    plain_start(p, STEP ? (const __nv_bfloat16*)x.q + t * x.ldq + v.qoff : (const __nv_bfloat16*)a.q + t * v.qstride + v.qoff, a.dim,
                MODE == UMBS_ATTN_SOFTMAX_SINK ? sink_score(a, v.h) : -INFINITY, MODE == UMBS_ATTN_SOFTMAX_SINK ? 1.f : 0.f);
    const int n_pool = STEP ? 0 : pooled_visible(rp, window, a.pool), lo = max(max(0, rp - window + 1), a.chunk > 0 ? rp / a.chunk * a.chunk : 0);
    bool go = true;
    for (int i = 0; go && i < n_pool; ++i) {
        const __nv_bfloat16* row = (const __nv_bfloat16*)a.pool_cache + ((int64_t)slot * a.pool_len + i) * v.row_kv;
        go = plain_key<MODE>(p, a, row + v.koff, a.dim, nullptr, row + v.voff, v.h, rp - i);
    }
    for (int j = lo; go && j <= rp; ++j) {
        if (STEP) {
            const int64_t key = start + j;
            go = plain_key<MODE>(p, a, (const __nv_bfloat16*)x.k + key * x.ldk + (int64_t)vh * x.kdim, x.kdim, (const __nv_bfloat16*)x.ks + key * x.ldks,
                                 (const __nv_bfloat16*)x.v + key * x.ldv + (int64_t)vh * a.vdim, v.h, rp - j);
        } else {
            const __nv_bfloat16* row = j >= pos0 ? (const __nv_bfloat16*)a.kv + (int64_t)(start + j - pos0) * v.row_kv
                                                 : (const __nv_bfloat16*)a.kv_cache + ((int64_t)slot * a.kv_len + j % a.kv_len) * v.row_kv;
            go = plain_key<MODE>(p, a, row + v.koff, a.dim, nullptr, row + v.voff, v.h, rp - j);
        }
    }
    const float inv = MODE == UMBS_ATTN_SIGMOID ? 1.f : 1.f / p.l;
    const float* grow = a.gate ? a.gate + t * a.ldg + (a.gate_per_head ? v.h : v.h * a.vdim) : nullptr;
    __nv_bfloat16* orow = STEP ? (__nv_bfloat16*)x.out + t * x.ldo + (int64_t)v.h * a.vdim : (__nv_bfloat16*)a.out + t * a.heads * a.vdim + (int64_t)v.h * a.vdim;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int c = lane + 32 * i;
        if (c < a.vdim) orow[c] = from_f32<__nv_bfloat16>(p.o[i] * inv * (grow ? sigmoidf_(grow[a.gate_per_head ? 0 : c]) : 1.f));
    }
}

// A gate's sigmoid.  The approximate reciprocal and one Newton-Raphson step are the rounded quotient for every 1 + e^-g below 2^126 (all of them compared); behind
// that come quotients below the smallest normal number, which the caller works out by the division (far).
__device__ __forceinline__ float gate_of(float g, bool& far) {
    const float x = 1.f + expf(-g), r = __fdividef(1.f, x);
    far |= x >= 0x1p126f;
    return fmaf(r, fmaf(-x, r, 1.f), r);
}

// 32 bytes, a whole sector of a thread's own row: with 16 at a time 4096 tokens, 16 heads of 128 over 4, take 100.3 us, so 97.9.
__device__ __forceinline__ void store32(void* p, const uint32_t* v) {
    asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]) : "memory");
}

template <int MODE, bool SHAPED, bool STEP>
__global__ void __launch_bounds__(kTaThreads, 2) attention_tc_kernel(const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_s, const __grid_constant__ CUtensorMap map_v,
                                                                        const __grid_constant__ CachedAttnArgs a, const __grid_constant__ StepKeys x, const __grid_constant__ Batch b, const TaDims z) {
    extern __shared__ unsigned char smem_raw[];
    __shared__ uint64_t bars[4 * kTaHeld + 8];
    __shared__ float s_row[2][2][kTaQ];                     // what a row's two threads tell each other: [tile parity][half]
    __shared__ uint32_t s_tmem;
    __shared__ int s_quit;
    uint64_t *k_full = bars, *k_empty = k_full + kTaHeld, *v_full = k_empty + kTaHeld, *v_empty = v_full + kTaHeld, *s_full = v_empty + kTaHeld, *p_full = s_full + 2,
             *o_full = s_full + 4, *q_full = s_full + 5, *lo_full = s_full + 6,        // (p_full: two in turn, a warp may be a tile ahead of another there)
             *v_landed = s_full + 7;                        // values of a last tile with rows behind the last
    volatile int* quit = &s_quit;
    if (threadIdx.x == 0) {
        for (int i = 0; i < kTaHeld; ++i) {
            umb::mbar_init(k_full + i, 2);
            umb::mbar_init(k_empty + i, 1);
            umb::mbar_init(v_full + i, 2);
            umb::mbar_init(v_empty + i, 1);
        }
        umb::mbar_init(s_full, 1);
        umb::mbar_init(s_full + 1, 1);
        umb::mbar_init(p_full, 8);
        umb::mbar_init(p_full + 1, 8);
        umb::mbar_init(o_full, 1);
        umb::mbar_init(q_full, 8);
        umb::mbar_init(lo_full, 8);
        umb::mbar_init(v_landed, 1);
        s_quit = 0;
        umb::fence_barrier_init();
    }
    chain_wait_only();
    // heads fastest, query tiles slowest and the last ones first: the blocks that see most keys start first, over all heads and sequences
    const int s = blockIdx.y, vh = blockIdx.x, q0 = (int)(gridDim.z - 1 - blockIdx.z) * kTaQ;
    const int len = b.seq_len[s], start = b.seq_start[s], pos0 = STEP ? 0 : b.seq_pos0[s], slot = STEP ? 0 : b.seq_slot[s];
    if (q0 >= len) return;
    VHead vhd;
    if (STEP) { vhd.h = vh; vhd.qoff = vh * a.dim; vhd.nv = a.heads; }
    else vhd = virtual_head(a, vh);
    const int h = vhd.h, window = a.window > 0 ? a.window : (1 << 30);
    const KeyTiles kt(a, window, pos0, q0, len);
    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
    const int k_bytes = z.q_atoms * (kTaK * 128), v_bytes = z.v_atoms * (kTaK * 128);
    unsigned char* smem = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    unsigned char* s_k = smem + z.q_atoms * (kTaQ * 128);   // Q [q_atoms][128 rows][128 B], tiles of K [q_atoms][64][128 B], of V [v_atoms][64][128 B]
    unsigned char* s_v = s_k + z.k_held * k_bytes;
    unsigned char* s_lo = s_v + z.v_held * v_bytes;         // third parts of the weights [128 rows][64 keys]

    if (warp == 8) {
        umb::tmem_alloc(&s_tmem, 256);
        umb::tmem_relinquish();
        chain_next();
    }
    umb::tc_fence_before();
    __syncthreads();
    umb::tc_fence_after();
    const uint32_t tmem = s_tmem;

    if (warp > 8) {
        // ------------------------------------------------------------------------------------ copies: 8 threads per 128-byte row piece
        const int tid = threadIdx.x - 288, ch = tid & 7, r0 = tid >> 3;
        const uint32_t sw = (uint32_t)((ch ^ (r0 & 7)) << 4);               // r0 + 8 p keeps r0's place inside its group of eight rows
        if (a.gate != nullptr && !a.gate_per_head)          // (read at the end, row by row)
            for (int e = tid; e < kTaQ * 4; e += 64)
                if (q0 + (e >> 2) < len && (e & 3) * 32 < a.vdim)
                    asm volatile("prefetch.global.L2 [%0];" ::"l"(a.gate + (int64_t)(start + q0 + (e >> 2)) * a.ldg + h * a.vdim + (e & 3) * 32));
        // A tile's keys go out before its values' place is waited for: the products that free it come behind this tile's scores.
        // Rows copied one by one are published when the next rows have been asked for, so that two groups are in flight; but keys at once
        // where there is one place for values, since the wait for it needs them.
        uint64_t* pending = nullptr;                        // asked for, not published
        auto publish = [&](bool all) {
            if (pending == nullptr) return;
            if (all) asm volatile("cp.async.wait_group 0;" ::: "memory");
            else asm volatile("cp.async.wait_group 1;" ::: "memory");
            umb::fence_proxy_async_smem();                  // this thread's copies are complete: show them to the tensor core
            __syncwarp();
            if (lane == 0) umb::mbar_arrive(pending);
            pending = nullptr;
        };
        auto asked = [&](uint64_t* bar) {
            asm volatile("cp.async.commit_group;" ::: "memory");
            publish(false);
            pending = bar;
        };
        int last_vs = -1;
        for (int i = 0; i < kt.n; ++i) {
            const int base = kt.base(i), last = kt.last(i), ks = i % z.k_held, vs = i % z.v_held;
            // rows that are neighbours: of the step (behind the last that a query sees come others', whose weights are 0: their scores are never looked at, their
            // values are cleared below; prompts of 20 tokens 13.3 us when those tiles were copied row by row), or of the ring where it does not begin again
            const int at0 = STEP ? 0 : base % a.kv_len;     // the first key's place in the ring
            const bool of_step = base >= pos0, of_ring = !STEP && base + kTaK <= pos0 && at0 + kTaK <= a.kv_len && (int64_t)(slot + 1) * a.kv_len <= z.ring_rows;
            const bool tma = z.tma && !kt.pooled(i) && (of_step || of_ring);
            const int row = of_step ? start + base - pos0 : (of_ring ? slot * a.kv_len + at0 : 0);
            // this thread's row p of four, 32 h behind the tile's first: where its keys and its values are (behind the last row: anywhere)
            auto row_of = [&](int h, int p, const __nv_bfloat16*& kp, const __nv_bfloat16*& vp) -> bool {
                const int j = base + r0 + 32 * h + 8 * p;
                const bool ok = j <= last;
                if (STEP) {
                    const int64_t t = start + (ok ? j : base);
                    kp = (const __nv_bfloat16*)x.k + t * x.ldk + (int64_t)vh * x.kdim;
                    vp = (const __nv_bfloat16*)x.v + t * x.ldv + (int64_t)vh * a.vdim;
                } else {
                    const __nv_bfloat16* row = (const __nv_bfloat16*)a.kv;
                    int place = at0 + j - base;
                    if (place >= a.kv_len) place = a.kv_len >= kTaK ? place - a.kv_len : j % a.kv_len;
                    if (ok)
                        row = kt.pooled(i) ? (const __nv_bfloat16*)a.pool_cache + ((int64_t)slot * a.pool_len + j) * vhd.row_kv
                            : j >= pos0 ? (const __nv_bfloat16*)a.kv + (int64_t)(start + j - pos0) * vhd.row_kv
                                        : (const __nv_bfloat16*)a.kv_cache + ((int64_t)slot * a.kv_len + place) * vhd.row_kv;
                    kp = row + vhd.koff;
                    vp = row + vhd.voff;
                }
                return ok;
            };
            bool free = true;
            if (i >= z.k_held) free = tc_spin_warp(k_empty + ks, (i / z.k_held - 1) & 1, quit);
            if (!__all_sync(0xffffffffu, free)) break;
            if (tma) {
                publish(true);
                if (umb::elect_one()) {
                    if (warp == 9) {
                        umb::mbar_arrive_expect_tx(k_full + ks, (uint32_t)k_bytes);
                        for (int at = 0; at < z.q_atoms; ++at) {
                            unsigned char* dst = s_k + ks * k_bytes + at * (kTaK * 128);
                            if (!STEP) tma_3d(dst, of_step ? &map_k : &map_s, vhd.koff + at * 64, row, 0, k_full + ks);
                            else if (at * 64 < x.kdim) tma_3d(dst, &map_k, vh * x.kdim + at * 64, row, 0, k_full + ks);
                            else tma_3d(dst, &map_s, at * 64 - x.kdim, row, 0, k_full + ks);
                        }
                    } else {
                        umb::mbar_arrive(k_full + ks);
                    }
                }
                __syncwarp();
            } else {
                for (int h = 0; h < 2; ++h)
#pragma unroll
                    for (int p = 0; p < 4; ++p) {
                        const __nv_bfloat16 *kp, *vp;
                        const bool in = row_of(h, p, kp, vp);
                        const uint32_t kd = smem_u32(s_k) + ks * k_bytes + (r0 + 32 * h + 8 * p) * 128 + sw;
                        for (int at = 0; at < z.q_atoms; ++at) {
                            const int d = at * 64 + ch * 8;
                            if (d >= z.k_steps * 16) continue;
                            const __nv_bfloat16* src = kp + d;                  // (a part all heads share follows a head's own)
                            if (STEP && d >= x.kdim) src = (const __nv_bfloat16*)x.ks + (int64_t)(start + (in ? base + r0 + 32 * h + 8 * p : base)) * x.ldks + (d - x.kdim);
                            const bool go = in && d < a.dim;
                            cp16(kd + at * (kTaK * 128), go ? src : kp, go ? 16 : 0);
                        }
                    }
                asked(k_full + ks);
                if (z.v_held == 1) publish(true);
            }
            if (i >= z.v_held) free = tc_spin_warp(v_empty + vs, (i / z.v_held - 1) & 1, quit);
            if (!__all_sync(0xffffffffu, free)) break;
            if (tma) {
                const bool clear = base + kTaK - 1 > last;  // (of the last tile alone)
                if (umb::elect_one()) {
                    if (warp == 10) {
                        uint64_t* bar = clear ? v_landed : v_full + vs;
                        umb::mbar_arrive_expect_tx(bar, (uint32_t)v_bytes);
                        for (int at = 0; at < z.v_atoms; ++at)
                            tma_3d(s_v + vs * v_bytes + at * (kTaK * 128), STEP || of_step ? &map_v : &map_s, (STEP ? vh * a.vdim : vhd.voff) + at * 64, row, 0, bar);
                    } else {
                        umb::mbar_arrive(v_full + vs);
                    }
                }
                __syncwarp();
                last_vs = clear ? vs : -1;
            } else {
                for (int h = 0; h < 2; ++h)
#pragma unroll
                    for (int p = 0; p < 4; ++p) {
                        const __nv_bfloat16 *kp, *vp;
                        const bool in = row_of(h, p, kp, vp);
                        const uint32_t vd = smem_u32(s_v) + vs * v_bytes + (r0 + 32 * h + 8 * p) * 128 + sw;
                        for (int at = 0; at < z.v_atoms; ++at) {
                            const int c = at * 64 + ch * 8;
                            const bool go = in && c < a.vdim;                   // rows that no query sees: zeros, their weights are 0
                            cp16(vd + at * (kTaK * 128), go ? vp + c : vp, go ? 16 : 0);
                        }
                    }
                asked(v_full + vs);
            }
        }
        publish(true);
        if (warp == 10 && last_vs >= 0 && tc_spin_warp(v_landed, 0, quit)) {
            const int rows = kt.last(kt.n - 1) - kt.base(kt.n - 1) + 1;
#pragma unroll 1
            for (int at = 0; at < z.v_atoms; ++at)
#pragma unroll 1
                for (int e = rows * 8 + lane; e < kTaK * 8; e += 32)
                    *reinterpret_cast<uint4*>(s_v + last_vs * v_bytes + at * (kTaK * 128) + e * 16) = make_uint4(0u, 0u, 0u, 0u);
            umb::fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) umb::mbar_arrive(v_full + last_vs);
        }
    } else if (warp == 8) {
        // ------------------------------------------------------------------------------------ products
        const uint32_t idesc_s = tc_idesc(kTaQ, kTaK), idesc_o = tc_idesc(kTaQ, 64, true) + ((z.v_atoms - 1) * (64u >> 3) << 17);
        const uint64_t qd = umb::umma_smem_desc_sw128(smem_u32(smem)), kd0 = umb::umma_smem_desc_sw128(smem_u32(s_k));
        // values: keys down the rows, so the operand is MN-major; its 64-wide pieces are 8192 bytes apart, groups of eight keys 1024
        const uint64_t vd0 = (umb::umma_smem_desc_sw128(smem_u32(s_v)) & ~((uint64_t)0x3fff << 16)) | ((uint64_t)(kTaK * 128 >> 4) << 16);
        const uint64_t ld = umb::umma_smem_desc_sw128(smem_u32(s_lo));
        // (the score columns of tile i held weights of tile i - 2, whose products are in front of these)
        auto scores = [&](int i, bool ready) -> bool {
            const int ks = i % z.k_held;
            if (!ready && !tc_spin_warp(k_full + ks, (i / z.k_held) & 1, quit)) return false;
            umb::tc_fence_after();
            const uint64_t kd = kd0 + ((ks * k_bytes) >> 4);
            if (umb::elect_one()) {
                for (int k = 0; k < z.k_steps; ++k)
                    umb::umma_ss_f16(tmem + (i & 1) * kTaK, qd + (k >> 2) * (kTaQ * 128 >> 4) + (k & 3) * 2, kd + (k >> 2) * (kTaK * 128 >> 4) + (k & 3) * 2,
                                     idesc_s, k ? 1u : 0u);
                umb::umma_commit(s_full + (i & 1));
                umb::umma_commit(k_empty + ks);
            }
            __syncwarp();
            return true;
        };
        bool ok = tc_spin_warp(q_full, 0, quit) && scores(0, false), k_ready = false;
        for (int i = 0; ok && i < kt.n; ++i) {
            const int vs = i % z.v_held;
            if (i + 1 < kt.n && !scores(i + 1, k_ready)) break;
            if (!tc_spin_warp(v_full + vs, (i / z.v_held) & 1, quit) || !tc_spin_warp(p_full + (i & 1), (i >> 1) & 1, quit)) break;
            umb::tc_fence_after();
            const uint64_t vd = vd0 + ((vs * v_bytes) >> 4);
            const uint32_t pt = tmem + (i & 1) * kTaK;
            if (umb::elect_one()) {
#pragma unroll
                for (int e = 0; e < 2; ++e)
#pragma unroll
                    for (int k = 0; k < kTaK / 16; ++k)
                        umb::umma_ts_f16(tmem + 128, pt + (k >> 1) * 32 + e * 16 + (k & 1) * 8, vd + k * (2048 >> 4), idesc_o, (i | e | k) ? 1u : 0u);
            }
            __syncwarp();
            if (!tc_spin_warp(lo_full, i & 1, quit)) break;
            const bool k_there = i + 2 < kt.n && tc_test(k_full + (i + 2) % z.k_held, ((i + 2) / z.k_held) & 1);
            umb::tc_fence_after();
            if (umb::elect_one()) {
#pragma unroll
                for (int k = 0; k < kTaK / 16; ++k) umb::umma_ss_f16(tmem + 128, ld + k * 2, vd + k * (2048 >> 4), idesc_o, 1u);
                umb::umma_commit(o_full);
                umb::umma_commit(v_empty + vs);
            }
            k_ready = __all_sync(0xffffffffu, k_there);
        }
    } else {
        // ------------------------------------------------------------------------------------ weights: two threads per row
        const int q = warp & 3, half = warp >> 2, row = q * 32 + lane;       // half: of a tile's keys, of the output's columns
        const int r = q0 + row, rp = pos0 + r;                              // the row's place in the step and its position
        const uint32_t t0 = tmem + ((uint32_t)(q * 32) << 16);
        constexpr float kLog2e = 1.4426950408889634f;
        const float c = SHAPED ? kLog2e : a.scale * kLog2e;
        const float hb = (MODE == UMBS_ATTN_SIGMOID && a.head_bias) ? a.head_bias[h] : 0.f;
        const float r1h = SHAPED && a.r1 ? a.r1[h] : 0.f, r2h = SHAPED && a.r1 ? a.r2[h] : 0.f;
        float m = MODE == UMBS_ATTN_SOFTMAX_SINK ? sink_score(a, h) * kLog2e : -INFINITY;      // the sink: a key of this score ...
        float l = MODE == UMBS_ATTN_SOFTMAX_SINK && half == 0 ? 1.f : 0.f;                     // ... without a value; the sum over this thread's keys
        const float gl = a.gate != nullptr && a.gate_per_head && r < len ? a.gate[(int64_t)(start + r) * a.ldg + h] : 0.f;
        const int tok_lo = max(rp - window + 1, a.chunk > 0 ? rp / a.chunk * a.chunk : 0);
        const int pool_hi = pooled_visible(rp, window, a.pool);
        {   // the queries: 8 threads per 128-byte row piece
            const int ch = threadIdx.x & 7, r0 = threadIdx.x >> 3;
            const __nv_bfloat16* qp = (const __nv_bfloat16*)(STEP ? x.q : a.q);
            const int64_t ldq = STEP ? x.ldq : vhd.qstride;
            for (int at = 0; at < z.q_atoms; ++at) {
                const int d = at * 64 + ch * 8;
                if (d >= z.k_steps * 16) continue;
#pragma unroll
                for (int p = 0; p < 4; ++p) {
                    const int qr = r0 + 32 * p;
                    const bool in = q0 + qr < len && d < a.dim;
                    cp16(smem_u32(smem) + at * (kTaQ * 128) + qr * 128 + ((ch ^ (qr & 7)) << 4), in ? qp + (int64_t)(start + q0 + qr) * ldq + vhd.qoff + d : qp, in ? 16 : 0);
                }
            }
            asm volatile("cp.async.wait_all;" ::: "memory");
            umb::fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) umb::mbar_arrive(q_full);
        }
        bool ok = true;
        for (int i = 0; i < kt.n; ++i) {
            const int base = kt.base(i) + 32 * half;        // keys base .. base + 31, of which [lo, hi) are visible to this row
            const int lo = kt.pooled(i) ? 0 : max(tok_lo - base, 0);
            const int hi = r >= len ? 0 : min((kt.pooled(i) ? pool_hi : rp + 1) - base, 32);
            const bool whole = __all_sync(0xffffffffu, lo == 0 && hi == 32);
            ok = tc_spin_warp(s_full + (i & 1), (i >> 1) & 1, quit);
            if (MODE == UMBS_ATTN_SIGMOID && !ok) break;    // (else both threads of a row leave at their barrier below)
            umb::tc_fence_after();
            uint32_t v[32];
            UMB_TMEM_LD_X32(t0 + (i & 1) * kTaK + half * 32, v);
            umb::tc_wait_ld();
            if (SHAPED) {
#pragma unroll
                for (int j = 0; j < 32; ++j) v[j] = __float_as_uint(shaped_score(a, __uint_as_float(v[j]), r1h, r2h, rp - (base + j)));
            }
            bool waited = i == 0;                           // the products of the tile before are done
            if (MODE != UMBS_ATTN_SIGMOID) {
                if (!whole) {
#pragma unroll
                    for (int j = 0; j < 32; ++j)
                        if (j < lo || j >= hi) v[j] = 0x7fffffffu;          // (a maximum passes a NaN by)
                }
                float m4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
                float mx;
                if (SHAPED || c > 0.f) {                    // (the product rounds every score alike: the largest stays the largest)
#pragma unroll
                    for (int j = 0; j < 32; ++j) m4[j & 3] = fmaxf(m4[j & 3], __uint_as_float(v[j]));
                    mx = fmaxf(fmaxf(m4[0], m4[1]), fmaxf(m4[2], m4[3])) * c;
                } else {
#pragma unroll
                    for (int j = 0; j < 32; ++j) m4[j & 3] = fmaxf(m4[j & 3], __uint_as_float(v[j]) * c);
                    mx = fmaxf(fmaxf(m4[0], m4[1]), fmaxf(m4[2], m4[3]));
                }
                s_row[i & 1][half][row] = mx;               // the larger of both threads'
                if (!(ok = pair_all(1 + q, ok))) break;
                mx = fmaxf(mx, s_row[i & 1][half ^ 1][row]);
                const bool move = mx > m + (i == 0 ? 0.f : kTaLazy) || (m == -INFINITY && mx > -INFINITY);
                if (__any_sync(0xffffffffu, move)) {        // rare behind the first tiles: the reference of some row moves
                    const float f = move ? ex2(m - mx) : 1.f;
                    if (move) m = mx;
                    l *= f;                                 // (m = -inf: l is 0)
                    if (i > 0) {
                        ok = tc_spin_warp(o_full, (i - 1) & 1, quit);
                        umb::tc_fence_after();
                        waited = true;
                        for (int c0 = half * 64; c0 < min(z.v_atoms * 64, half * 64 + 64); c0 += 16) {
                            uint32_t o[16];
                            UMB_TMEM_LD_X16(t0 + 128 + c0, o);
                            umb::tc_wait_ld();
#pragma unroll
                            for (int j = 0; j < 16; ++j) o[j] = __float_as_uint(__uint_as_float(o[j]) * f);
                            UMB_TMEM_ST_X16(t0 + 128 + c0, o);
                        }
                    }
                }
            }
            const float ref = m == -INFINITY ? 0.f : m;
            // two numbers an instruction where there is one for two
            if (MODE == UMBS_ATTN_SIGMOID) {
#pragma unroll
                for (int j = 0; j < 32; ++j) v[j] = __float_as_uint(sigmoidf_(__uint_as_float(v[j]) * a.scale + hb));
            } else {
                const f32x2 cc = pack2(c, c), rr = pack2(-ref, -ref);
#pragma unroll
                for (int j = 0; j < 32; j += 2) {
                    const float2 z = unpack2(fma2(pack2(__uint_as_float(v[j]), __uint_as_float(v[j + 1])), cc, rr));
                    v[j] = __float_as_uint(ex2(z.x));
                    v[j + 1] = __float_as_uint(ex2(z.y));
                }
            }
            if (!whole) {
#pragma unroll
                for (int j = 0; j < 32; ++j)
                    if (j < lo || j >= hi) v[j] = 0u;
            }
            // the three parts, one after the other; what is left of a weight stays in its place.  The products of the first two begin while the
            // third waits for its place, which the products of the tile before read.
            f32x2 l2[2] = {0ull, 0ull};
#pragma unroll
            for (int e = 0; e < 3; ++e) {
                uint32_t ph[16];
#pragma unroll
                for (int j = 0; j < 16; ++j) {
                    const float p = __uint_as_float(v[2 * j]), p1 = __uint_as_float(v[2 * j + 1]);
                    ph[j] = hi_pair(p, p1);
                    if (e == 2) continue;
                    const f32x2 pp = pack2(p, p1);
                    if (e == 0) l2[j & 1] = add2(l2[j & 1], pp);
                    const float2 left = unpack2(add2(pp, pack2(minus_cut(p), minus_cut(p1))));
                    v[2 * j] = __float_as_uint(left.x);
                    v[2 * j + 1] = __float_as_uint(left.y);
                }
                if (e < 2) UMB_TMEM_ST_X16(t0 + (i & 1) * kTaK + half * 32 + e * 16, ph);
                if (e == 1) {
                    umb::tc_wait_st();
                    umb::tc_fence_before();
                    __syncwarp();
                    if (lane == 0) umb::mbar_arrive(p_full + (i & 1));
                }
                if (e == 2) {
                    if (!waited) ok = tc_spin_warp(o_full, (i - 1) & 1, quit);
#pragma unroll
                    for (int c = 0; c < 4; ++c)
                        *reinterpret_cast<uint4*>(s_lo + row * 128 + (((half * 4 + c) ^ (row & 7)) << 4)) = make_uint4(ph[4 * c], ph[4 * c + 1], ph[4 * c + 2], ph[4 * c + 3]);
                    umb::fence_proxy_async_smem();
                    __syncwarp();
                    if (lane == 0) umb::mbar_arrive(lo_full);
                }
            }
            const float2 la = unpack2(l2[0]), lb = unpack2(l2[1]);
            l += (la.x + la.y) + (lb.x + lb.y);
        }
        // both threads' sums (also where a wait was given up: the other warp may be at this barrier)
        ok = ok && tc_spin_warp(o_full, (kt.n - 1) & 1, quit);
        s_row[kt.n & 1][half][row] = l;
        pair_sync(1 + q);
        l = s_row[kt.n & 1][0][row] + s_row[kt.n & 1][1][row];
        // Results with a gate per column go through shared memory (everything in it has been used), so that gates and outputs are whole pieces of rows: a
        // thread's own row of both is 12 us of a block's 60.  Others go straight from the registers, half a row a thread: prompts of 77 tokens, heads of 64, 8.4 us
        // through shared memory, 7.9 like this.
        float* s_o = reinterpret_cast<float*>(smem);
        const int ldo = z.v_atoms * 64 + 4;                 // (rows four banks apart)
        const bool gates = a.gate != nullptr && !a.gate_per_head;
        const int64_t ldout = STEP ? x.ldo : (int64_t)a.heads * a.vdim;
        float odd = 0.f;                                    // stays 0 while the row's sums are finite
        if (ok) {
            umb::tc_fence_after();
            const float inv = MODE == UMBS_ATTN_SIGMOID ? 1.f : 1.f / l;
            const float gh = a.gate != nullptr && a.gate_per_head && r < len ? sigmoidf_(gl) : 1.f;
            for (int c0 = half * 64; c0 < min(a.vdim, half * 64 + 64); c0 += 32) {
                uint32_t v[32];
                UMB_TMEM_LD_X32(t0 + 128 + c0, v);
                umb::tc_wait_ld();
#pragma unroll
                for (int e = 0; e < 32; e += 4) {
                    float4 o;
                    o.x = __uint_as_float(v[e]) * inv;
                    o.y = __uint_as_float(v[e + 1]) * inv;
                    o.z = __uint_as_float(v[e + 2]) * inv;
                    o.w = __uint_as_float(v[e + 3]) * inv;
                    if (r < len && c0 + e < a.vdim) odd = fmaf(o.w, 0.f, fmaf(o.z, 0.f, fmaf(o.y, 0.f, fmaf(o.x, 0.f, odd))));
                    if (gates) *reinterpret_cast<float4*>(s_o + row * ldo + c0 + e) = o;
                    else {
                        const __nv_bfloat162 w0 = __floats2bfloat162_rn(o.x * gh, o.y * gh), w1 = __floats2bfloat162_rn(o.z * gh, o.w * gh);
                        v[e >> 1] = *reinterpret_cast<const uint32_t*>(&w0);
                        v[(e >> 1) + 1] = *reinterpret_cast<const uint32_t*>(&w1);
                    }
                }
                if (!gates && r < len) {
                    uint4* orow = reinterpret_cast<uint4*>((__nv_bfloat16*)(STEP ? x.out : a.out) + (start + r) * ldout + (int64_t)h * a.vdim + c0);
                    if (((uintptr_t)orow & 31) == 0 && c0 + 32 <= a.vdim) {
                        store32(orow, &v[0]);
                        store32(orow + 2, &v[8]);
                    } else {
#pragma unroll
                        for (int e = 0; e < 4; ++e)
                            if (c0 + 8 * e < a.vdim) orow[e] = make_uint4(v[4 * e], v[4 * e + 1], v[4 * e + 2], v[4 * e + 3]);
                    }
                }
            }
        }
        s_row[(kt.n & 1) ^ 1][half][row] = odd;
        if (!pair_all(5 + q, ok)) ok = false;
        if (ok && gates) {
            // this warp's half of the quarter's rows, 4 columns a lane, eight rows' gates at a time
            const int c = lane * 4, row0 = q * 32 + half * 16;
            __nv_bfloat16* op = (__nv_bfloat16*)(STEP ? x.out : a.out) + (int64_t)h * a.vdim + c;
            // (loops rather than one long stretch: each instruction of a short prompt's block is fetched for it alone)
            auto put = [&](int orow, float4 o) {
                const __nv_bfloat162 w0 = __floats2bfloat162_rn(o.x, o.y), w1 = __floats2bfloat162_rn(o.z, o.w);
                *reinterpret_cast<uint2*>(op + (int64_t)(start + q0 + orow) * ldout) = make_uint2(*reinterpret_cast<const uint32_t*>(&w0), *reinterpret_cast<const uint32_t*>(&w1));
            };
            const int rows = c < a.vdim ? min(16, len - q0 - row0) : 0;
#pragma unroll 1
            for (int e0 = 0; e0 < rows; e0 += 8) {
                float4 g[8];
#pragma unroll
                for (int e = 0; e < 8; ++e)
                    if (e0 + e < rows) {
                        const float* gp = a.gate + (int64_t)(start + q0 + row0 + e0 + e) * a.ldg + h * a.vdim + c;
                        g[e] = ((uintptr_t)gp & 15) == 0 ? *reinterpret_cast<const float4*>(gp) : make_float4(gp[0], gp[1], gp[2], gp[3]);
                    }
                bool far = false;
#pragma unroll
                for (int e = 0; e < 8; ++e)
                    if (e0 + e < rows) {
                        const float4 o = *reinterpret_cast<const float4*>(s_o + (row0 + e0 + e) * ldo + c);
                        const float4 w = make_float4(gate_of(g[e].x, far), gate_of(g[e].y, far), gate_of(g[e].z, far), gate_of(g[e].w, far));
                        put(row0 + e0 + e, make_float4(o.x * w.x, o.y * w.y, o.z * w.z, o.w * w.w));
                    }
                if (far) {                              // rare: these rows once more
#pragma unroll 1
                    for (int e = e0; e < min(rows, e0 + 8); ++e) {
                        const float* gp = a.gate + (int64_t)(start + q0 + row0 + e) * a.ldg + h * a.vdim + c;
                        const float4 o = *reinterpret_cast<const float4*>(s_o + (row0 + e) * ldo + c);
                        put(row0 + e, make_float4(o.x * sigmoidf_(gp[0]), o.y * sigmoidf_(gp[1]), o.z * sigmoidf_(gp[2]), o.w * sigmoidf_(gp[3])));
                    }
                }
            }
        }
        // a row that is odd in either half: by the first half's warp, when both have stored theirs
        pair_sync(5 + q);
        if (ok && half == 0)
            for (uint32_t rows = __ballot_sync(0xffffffffu, s_row[(kt.n & 1) ^ 1][0][row] != 0.f || s_row[(kt.n & 1) ^ 1][1][row] != 0.f); rows != 0; rows &= rows - 1)
                plain_row<MODE, STEP>(a, x, b, s, vh, q0 + q * 32 + __ffs(rows) - 1);
    }
    __syncwarp();
    umb::tc_fence_before();
    __syncthreads();
    tc_settle(quit, z.report);
    if (warp == 8) {
        umb::tc_fence_after();
        umb::tmem_dealloc(tmem, 256);
    }
}

// Two key tiles and two value tiles where that leaves room for a second block on the SM (228 KB, 1 KB of it per block the system's): one key tile beside
// queries of more than 64 numbers (the next one comes while weights are made), and one value tile beside more than 128.
constexpr int kTaTiles = 110 * 1024, kTaSmem = 1024 + kTaTiles;     // the largest of them
static int ta_smem(const TaDims& z) { return 1024 + (z.q_atoms * (kTaQ + z.k_held * kTaK) + z.v_held * z.v_atoms * kTaK + kTaQ) * 128; }
static TaDims ta_dims(const CachedAttnArgs& a) {
    TaDims z{(a.dim + 63) / 64, (a.dim + 15) / 16, (a.vdim + 63) / 64, kTaHeld, kTaHeld, 0, 0, nullptr};
    if (ta_smem(z) > kTaSmem) z.k_held = 1;
    if (ta_smem(z) > kTaSmem) z.v_held = 1;
    return z;
}

// Every row piece is copied in 16-byte pieces and a block's tiles and tensor memory leave room for a second one on the SM:
// sizes in eights, queries and keys of up to 192, values of up to 128 numbers.
// bf16 results only: the tensor core cuts its running sums off instead of rounding them, which leaves an fp32 result 1.2e-6
// from float64 (in the norm, 600 keys) where the fp32 kernel leaves 4e-7, so results handed out in fp32 keep that kernel.
bool attention_tc_fits(const CachedAttnArgs& a, const StepKeys* s) {
    if (s == nullptr && a.raw != nullptr) return false;
    auto al = [](const void* p) { return ((uintptr_t)p & 15) == 0; };
    if (a.dim % 8 || a.vdim % 8 || a.dim > 192 || a.vdim > 128 || a.dim < 8 || a.vdim < 8) return false;
    if (s != nullptr)
        return s->kdim % 8 == 0 && al(s->q) && al(s->k) && al(s->v) && al(s->out) && s->ldq % 8 == 0 && s->ldk % 8 == 0 && s->ldv % 8 == 0 &&
               s->ldo % 8 == 0 && (s->kdim == a.dim || (al(s->ks) && s->ldks % 8 == 0));
    return al(a.q) && al(a.kv) && al(a.kv_cache) && (a.pool <= 0 || al(a.pool_cache)) && al(a.out);
}

// from p to the end of the allocation that it points into; 0 where that is not known
static uint64_t bytes_from(const void* p) {
    typedef CUresult (*AddressRange)(CUdeviceptr*, size_t*, CUdeviceptr);
    static const AddressRange fn = [] {
        void* sym = nullptr;
        cudaDriverEntryPointQueryResult q;
        return cudaGetDriverEntryPoint("cuMemGetAddressRange", &sym, cudaEnableDefault, &q) == cudaSuccess && q == cudaDriverEntryPointSuccess ? (AddressRange)sym
                                                                                                                                            : nullptr;
    }();
    CUdeviceptr base = 0;
    size_t size = 0;
    if (fn == nullptr || fn(&base, &size, (CUdeviceptr)p) != CUDA_SUCCESS || (CUdeviceptr)p < base) return 0;
    return base + size - (CUdeviceptr)p;
}

template <int MODE, bool SHAPED, bool STEP>
static int launch_ta(const CachedAttnArgs& a, const StepKeys& x, const Batch& b, cudaStream_t st) {
    TaDims z = ta_dims(a);
    int rc = give_up_word(&z.report);
    if (rc == 0) rc = give_up_status();
    if (rc != 0) return rc;
    // Rows as tensor maps: the step's, and of a cache the ring's (map_s).  Columns behind a head's own in its last piece of 64 are never used: products end
    // with the head's k steps (of 16: behind an odd multiple of 8 they meet zeros of the query), and output columns are the head's.  A part that all heads share
    // begins behind whole pieces.  Rows that overlap (a row repeated among them) and whatever else a map does not describe are copied row by row.
    CUtensorMap mk{}, ms{}, mv{};
    z.tma = !STEP || ((x.kdim % 64 == 0 || x.kdim == a.dim) && x.ldk >= (int64_t)a.heads * x.kdim && x.ldv >= (int64_t)a.heads * a.vdim &&
                      (x.kdim == a.dim || x.ldks >= a.dim - x.kdim));
    if (z.tma) {
        if (STEP) {
            rc = encode_map(&mk, x.k, (uint64_t)a.heads * x.kdim, b.n_tokens, 1, x.ldk, 0, kTaK);
            if (rc == 0 && x.kdim < a.dim) rc = encode_map(&ms, x.ks, a.dim - x.kdim, b.n_tokens, 1, x.ldks, 0, kTaK);
            if (rc == 0) rc = encode_map(&mv, x.v, (uint64_t)a.heads * a.vdim, b.n_tokens, 1, x.ldv, 0, kTaK);
        } else {
            // (how many slots the caller's cache has is not known here: the map ends with the memory that the cache is in)
            const uint64_t row = (uint64_t)a.kv_heads * ((a.maps > 1 ? a.maps : 1) * a.dim + a.vdim);
            z.ring_rows = (int64_t)std::min<uint64_t>({0x7fffffff, (1ull << 38) / row, bytes_from(a.kv_cache) / (row * 2)});
            rc = encode_map(&mk, a.kv, row, b.n_tokens, 1, row, 0, kTaK);
            if (rc == 0 && z.ring_rows > 0) rc = encode_map(&ms, a.kv_cache, row, z.ring_rows, 1, row, 0, kTaK);
            mv = mk;
        }
        z.tma = rc == 0;
    }
    const int smem = ta_smem(z);
    auto kernel = attention_tc_kernel<MODE, SHAPED, STEP>;
    // (always the same limit: another thread may be between setting it and its launch)
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kTaSmem);
    if (e != cudaSuccess) return (int)e;
    return chain_launch(kernel, dim3(a.heads, b.n_seqs, (b.max_seq_len + kTaQ - 1) / kTaQ), kTaThreads, smem, st, mk, ms, mv, a, x, b, z);
}

int launch_attention_tc(int mode, const CachedAttnArgs& a, const StepKeys* keys, const Batch& b, cudaStream_t st) {
    const bool shaped = a.softcap > 0.f || a.r1 != nullptr;
    if (keys != nullptr)
        return mode == UMBS_ATTN_SOFTMAX_SINK ? launch_ta<UMBS_ATTN_SOFTMAX_SINK, false, true>(a, *keys, b, st)
                                              : launch_ta<UMBS_ATTN_SOFTMAX, false, true>(a, *keys, b, st);
    const StepKeys none{};
    switch (mode) {
        case UMBS_ATTN_SOFTMAX:
            return shaped ? launch_ta<UMBS_ATTN_SOFTMAX, true, false>(a, none, b, st) : launch_ta<UMBS_ATTN_SOFTMAX, false, false>(a, none, b, st);
        case UMBS_ATTN_SOFTMAX_SINK:
            return shaped ? launch_ta<UMBS_ATTN_SOFTMAX_SINK, true, false>(a, none, b, st) : launch_ta<UMBS_ATTN_SOFTMAX_SINK, false, false>(a, none, b, st);
        case UMBS_ATTN_SIGMOID: return launch_ta<UMBS_ATTN_SIGMOID, false, false>(a, none, b, st);
    }
    return UMB_ERR_ARG;
}

unsigned int attention_tc_timeouts() { return tc_timeouts(); }

}  // namespace umbs
