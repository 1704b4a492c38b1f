// Attention of a step with several tokens per sequence on the 5th-generation tensor cores, bf16 storage: the tile kernels of
// seq_cached_attn.cu and seq_window_attn.cu for the sizes and addresses it takes.
//
// A block = 128 consecutive query rows of one (sequence, head) = the 128 lanes of tensor memory; two blocks share an
// SM.  Tiles of 32 keys run through three stages that overlap:
//   warps 5-6  bring key and value rows into the 128-byte-swizzled images the tensor core reads, several tiles ahead: with TMA
//              where the 32 rows are neighbours in the step and heads are whole pieces of 64 numbers, else with 16-byte
//              cp.async, each row from where it lives (step, ring, block table), zeros where there is none;
//   warp 4     one thread issues S = Q K^T of the next tile, then O += P V of this one, accumulators in tensor memory;
//   warps 0-3  a thread per row: scores to weights in fp32 in the base-2 domain, an online reference that only moves when a
//              score passes it by 2^8 (then O is rescaled), the row's sum.
// Weights stay 32-bit: an fp32 weight is the sum of three bf16 numbers (8 + 8 + 8 significant bits, cut off one after the
// other, so exactly), and P V is three products against the same values.  Products of bf16 operands are exact in the tensor
// core and its sums are fp32.
//
// Tensor memory, 256 columns: two score tiles 0-31 and 32-63, the weights' parts 64-79, 80-95, 96-111, output 128-255.  With
// 64 keys to a tile only one score tile fits beside the output of 128 columns, and scores, weights and output products take
// turns: 5800 clocks per 64 keys and block, of which the tensor core works 1160 (measured with clock64 stamps; 128 x 64 x 16
// takes it 48 clocks, 128 x 128 x 16 takes 64).
//
// Bound: the weights (an exponential and three bf16 parts of each score by the row's own thread: 1450 of a tile's 2400 clocks) beside
// products of 32 keys, and blocks that fill the SMs 1.7 times.  4096 tokens, 16 heads of 128 over 4 key/value heads, window 1024, pooled
// blocks: 2250 us on fp32 multiply-adds, 141 with waits of 330 clocks for barriers that were through, 115 here; two prompts of 2000
// tokens, 16 heads of 128 + 64 shared: 2652 -> 188 -> 158 us.
#include "seq_attn.h"
#include "seq_tc.cuh"

namespace umbs {

constexpr int kTaQ = 128, kTaK = 32;
constexpr int kTaThreads = 224;                             // 4 warps of weights, 1 of products, 2 of copies
constexpr int kTaStages = 4;                                // key and value tiles held, at most
constexpr float kTaLazy = 8.f;                              // how far (in powers of two) a score may pass the reference

// 64-wide pieces of a query row, 16-wide k steps, 64-wide pieces of a value row; tiles held; give_up_word()
struct TaDims { int q_atoms, k_steps, v_atoms, stages, tma; unsigned int* report; };

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

template <int MODE, bool SHAPED, bool STEP>
__global__ void __launch_bounds__(kTaThreads, 2) attention_tc_kernel(const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_s, const __grid_constant__ CUtensorMap map_v,
                                                                        const __grid_constant__ CachedAttnArgs a, const __grid_constant__ StepKeys x, const __grid_constant__ Batch b, const TaDims z) {
    extern __shared__ unsigned char smem_raw[];
    __shared__ uint64_t bars[4 * kTaStages + 4];
    __shared__ uint32_t s_tmem;
    __shared__ int s_quit;
    uint64_t *k_full = bars, *v_full = bars + kTaStages, *k_empty = bars + 2 * kTaStages, *v_empty = bars + 3 * kTaStages,
             *s_full = bars + 4 * kTaStages, *p_full = s_full + 2, *o_full = s_full + 3;
    volatile int* quit = &s_quit;
    chain_wait_only();
    const int s = blockIdx.z, vh = blockIdx.y, q0 = (int)(gridDim.x - 1 - blockIdx.x) * kTaQ;     // the rows that see most start first
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
    unsigned char* s_k = smem + z.q_atoms * (kTaQ * 128);   // Q [q_atoms][128 rows][128 B], stages of K [q_atoms][32][128 B], of V [v_atoms][32][128 B]
    unsigned char* s_v = s_k + z.stages * k_bytes;

    if (threadIdx.x == 0) {
        for (int i = 0; i < kTaStages; ++i) {
            umb::mbar_init(k_full + i, 2);
            umb::mbar_init(v_full + i, 2);
            umb::mbar_init(k_empty + i, 1);
            umb::mbar_init(v_empty + i, 1);
        }
        umb::mbar_init(s_full, 1);
        umb::mbar_init(s_full + 1, 1);
        umb::mbar_init(p_full, 4);
        umb::mbar_init(o_full, 1);
        s_quit = 0;
        umb::fence_barrier_init();
    }
    if (warp == 4) {
        umb::tmem_alloc(&s_tmem, 256);
        umb::tmem_relinquish();
        chain_next();
    }
    umb::tc_fence_before();
    __syncthreads();
    umb::tc_fence_after();
    const uint32_t tmem = s_tmem;

    if (warp > 4) {
        // ------------------------------------------------------------------------------------ copies: 8 threads per 128-byte row piece
        const int tid = threadIdx.x - 160, ch = tid & 7, r0 = tid >> 3, stages = z.stages;
        const uint32_t sw = (uint32_t)((ch ^ (r0 & 7)) << 4);               // r0 + 8 p keeps r0's place inside its group of eight rows
        const __nv_bfloat16* q = (const __nv_bfloat16*)(STEP ? x.q : a.q);
        const int64_t ldq = STEP ? x.ldq : vhd.qstride;
        for (int at = 0; at < z.q_atoms; ++at) {
            const int d = at * 64 + ch * 8;
            if (d >= z.k_steps * 16) continue;
#pragma unroll 4
            for (int p = 0; p < 16; ++p) {
                const int r = r0 + 8 * p;
                const bool in = q0 + r < len && d < a.dim;
                cp16(smem_u32(smem) + at * (kTaQ * 128) + r * 128 + sw, in ? q + (int64_t)(start + q0 + r) * ldq + vhd.qoff + d : q, in ? 16 : 0);
            }
        }
        // A tile's copies are published when the tile behind it has been asked for: two are in flight.  (Publishing waits for the
        // stage of that next tile, which is free long before: there are three stages or four.)
        auto publish = [&](int i) {
            umb::fence_proxy_async_smem();                  // this thread's copies are complete: show them to the tensor core
            __syncwarp();
            if (lane == 0) {
                umb::mbar_arrive(k_full + i % stages);
                umb::mbar_arrive(v_full + i % stages);
            }
        };
        int i = 0, pending = 0;                             // pending: the tile before has been asked for but not published
        for (; i < kt.n; ++i) {
            const int base = kt.base(i), last = kt.last(i), st = i % stages;
            bool free = true;
            if (i >= stages) free = tc_poll(k_empty + st, (i / stages - 1) & 1, quit) && tc_poll(v_empty + st, (i / stages - 1) & 1, quit);
            if (!__all_sync(0xffffffffu, free)) break;
            if (z.tma && !kt.pooled(i) && base >= pos0 && base + kTaK - 1 <= last) {
                if (i == 0 || pending) {                    // (the queries come with the first tile)
                    asm volatile("cp.async.wait_all;" ::: "memory");
                    if (pending) publish(i - 1);
                    else umb::fence_proxy_async_smem();
                    __syncwarp();
                    pending = 0;
                }
                if (umb::elect_one()) {
                    const int row = start + base - pos0;
                    if (warp == 5) {
                        umb::mbar_arrive_expect_tx(k_full + st, (uint32_t)k_bytes);
                        for (int at = 0; at < z.q_atoms; ++at) {
                            unsigned char* dst = s_k + st * k_bytes + at * (kTaK * 128);
                            if (!STEP) tma_3d(dst, &map_k, vhd.koff + at * 64, row, 0, k_full + st);
                            else if (at * 64 < x.kdim) tma_3d(dst, &map_k, vh * x.kdim + at * 64, row, 0, k_full + st);
                            else tma_3d(dst, &map_s, at * 64 - x.kdim, row, 0, k_full + st);
                        }
                        umb::mbar_arrive(v_full + st);
                    } else {
                        umb::mbar_arrive_expect_tx(v_full + st, (uint32_t)v_bytes);
                        for (int at = 0; at < z.v_atoms; ++at)
                            tma_3d(s_v + st * v_bytes + at * (kTaK * 128), &map_v, (STEP ? vh * a.vdim : vhd.voff) + at * 64, row, 0, v_full + st);
                        umb::mbar_arrive(k_full + st);
                    }
                }
                __syncwarp();
                continue;
            }
            const __nv_bfloat16 *kp[4], *vp[4];             // this thread's rows: keys, values
            uint32_t in = 0;
#pragma unroll
            for (int p = 0; p < 4; ++p) {
                const int j = base + r0 + 8 * p;
                const bool ok = j <= last;
                in |= (uint32_t)ok << p;
                if (STEP) {
                    const int64_t t = start + (ok ? j : base);
                    kp[p] = (const __nv_bfloat16*)x.k + t * x.ldk + (int64_t)vh * x.kdim;
                    vp[p] = (const __nv_bfloat16*)x.v + t * x.ldv + (int64_t)vh * a.vdim;
                } else {
                    const __nv_bfloat16* row = (const __nv_bfloat16*)a.kv;
                    if (ok)
                        row = kt.pooled(i) ? (const __nv_bfloat16*)a.pool_cache + ((int64_t)slot * a.pool_len + j) * vhd.row_kv
                            : j >= pos0 ? (const __nv_bfloat16*)a.kv + (int64_t)(start + j - pos0) * vhd.row_kv
                                        : (const __nv_bfloat16*)a.kv_cache + ((int64_t)slot * a.kv_len + j % a.kv_len) * vhd.row_kv;
                    kp[p] = row + vhd.koff;
                    vp[p] = row + vhd.voff;
                }
            }
            const uint32_t kd = smem_u32(s_k) + st * k_bytes + r0 * 128 + sw, vd = smem_u32(s_v) + st * v_bytes + r0 * 128 + sw;
            for (int at = 0; at < z.q_atoms; ++at) {
                const int d = at * 64 + ch * 8;
                if (d >= z.k_steps * 16) continue;
                const bool own = !STEP || d < x.kdim, dok = d < a.dim;      // (a part all heads share follows a head's own)
#pragma unroll
                for (int p = 0; p < 4; ++p) {
                    const __nv_bfloat16* src = kp[p] + d;
                    if (STEP && !own) src = (const __nv_bfloat16*)x.ks + (int64_t)(start + ((in >> p & 1) ? base + r0 + 8 * p : base)) * x.ldks + (d - x.kdim);
                    const bool go = (in >> p & 1) && dok;
                    cp16(kd + at * (kTaK * 128) + p * 1024, go ? src : kp[p], go ? 16 : 0);
                }
            }
            for (int at = 0; at < z.v_atoms; ++at) {
                const int c = at * 64 + ch * 8;
#pragma unroll
                for (int p = 0; p < 4; ++p) {
                    const bool go = (in >> p & 1) && c < a.vdim;            // rows that no query sees: zeros, their weights are 0
                    cp16(vd + at * (kTaK * 128) + p * 1024, go ? vp[p] + c : vp[p], go ? 16 : 0);
                }
            }
            asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 1;" ::: "memory");
            if (pending) publish(i - 1);
            pending = 1;
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        if (i == kt.n && pending) publish(kt.n - 1);
    } else if (warp == 4) {
        // ------------------------------------------------------------------------------------ products
        const uint32_t idesc_s = tc_idesc(kTaQ, kTaK), idesc_o = tc_idesc(kTaQ, 64, true) + ((z.v_atoms - 1) * (64u >> 3) << 17);
        const uint64_t qd = umb::umma_smem_desc_sw128(smem_u32(smem)), kd0 = umb::umma_smem_desc_sw128(smem_u32(s_k));
        // values: keys down the rows, so the operand is MN-major; its 64-wide pieces are 4096 bytes apart, groups of eight keys 1024
        const uint64_t vd0 = (umb::umma_smem_desc_sw128(smem_u32(s_v)) & ~((uint64_t)0x3fff << 16)) | ((uint64_t)(kTaK * 128 >> 4) << 16);
        auto scores = [&](int i, bool ready) -> bool {      // the tile's score columns were read two tiles ago, in front of weights already waited for
            const int st = i % z.stages;
            if (!ready && !tc_spin_warp(k_full + st, (i / z.stages) & 1, quit)) return false;
            umb::tc_fence_after();
            const uint64_t kd = kd0 + ((st * k_bytes) >> 4);
            if (umb::elect_one()) {
                for (int k = 0; k < z.k_steps; ++k)
                    umb::umma_ss_f16(tmem + (i & 1) * kTaK, qd + (k >> 2) * (kTaQ * 128 >> 4) + (k & 3) * 2, kd + (k >> 2) * (kTaK * 128 >> 4) + (k & 3) * 2,
                                     idesc_s, k ? 1u : 0u);
                umb::umma_commit(s_full + (i & 1));
                umb::umma_commit(k_empty + st);
            }
            __syncwarp();
            return true;
        };
        bool ok = scores(0, false), k_ready = false;
        for (int i = 0; ok && i < kt.n; ++i) {
            const int st = i % z.stages;
            const bool v_there = tc_test(v_full + st, (i / z.stages) & 1);
            if (i + 1 < kt.n && !scores(i + 1, k_ready)) break;
            if (!__all_sync(0xffffffffu, v_there) && !tc_spin_warp(v_full + st, (i / z.stages) & 1, quit)) break;
            if (!tc_spin_warp(p_full, i & 1, quit)) break;
            const bool k_there = i + 2 < kt.n && tc_test(k_full + (i + 2) % z.stages, ((i + 2) / z.stages) & 1);
            umb::tc_fence_after();
            const uint64_t vd = vd0 + ((st * v_bytes) >> 4);
            if (umb::elect_one()) {
#pragma unroll
                for (int e = 0; e < 3; ++e)
#pragma unroll
                    for (int k = 0; k < kTaK / 16; ++k)
                        umb::umma_ts_f16(tmem + 128, tmem + 64 + e * 16 + k * 8, vd + k * (2048 >> 4), idesc_o, (i | e | k) ? 1u : 0u);
                umb::umma_commit(o_full);
                umb::umma_commit(v_empty + st);
            }
            k_ready = __all_sync(0xffffffffu, k_there);
        }
    } else {
        // ------------------------------------------------------------------------------------ weights: a thread per row
        const int r = q0 + warp * 32 + lane, rp = pos0 + r;                 // the row's place in the step and its position
        const uint32_t t0 = tmem + ((uint32_t)(warp * 32) << 16);
        constexpr float kLog2e = 1.4426950408889634f;
        const float c = SHAPED ? kLog2e : a.scale * kLog2e;
        const float hb = (MODE == UMBS_ATTN_SIGMOID && a.head_bias) ? a.head_bias[h] : 0.f;
        const float r1h = SHAPED && a.r1 ? a.r1[h] : 0.f, r2h = SHAPED && a.r1 ? a.r2[h] : 0.f;
        float m = MODE == UMBS_ATTN_SOFTMAX_SINK ? sink_score(a, h) * kLog2e : -INFINITY;      // the sink: a key of this score ...
        float l = MODE == UMBS_ATTN_SOFTMAX_SINK ? 1.f : 0.f;                                  // ... without a value
        const int tok_lo = max(rp - window + 1, a.chunk > 0 ? rp / a.chunk * a.chunk : 0);
        const int pool_hi = pooled_visible(rp, window, a.pool);
        bool ok = true, s_ready = false;
        for (int i = 0; i < kt.n; ++i) {
            const int base = kt.base(i);                    // keys base .. base + 31, of which [lo, hi) are visible to this row
            const int lo = kt.pooled(i) ? 0 : max(tok_lo - base, 0);
            const int hi = r >= len ? 0 : min((kt.pooled(i) ? pool_hi : rp + 1) - base, kTaK);
            const bool whole = __all_sync(0xffffffffu, lo == 0 && hi == kTaK);
            if (!s_ready && !(ok = tc_spin_warp(s_full + (i & 1), (i >> 1) & 1, quit))) break;
            umb::tc_fence_after();
            uint32_t v[32];
            UMB_TMEM_LD_X32(t0 + (i & 1) * kTaK, v);
            umb::tc_wait_ld();
            if (SHAPED) {
#pragma unroll
                for (int j = 0; j < 32; ++j) v[j] = __float_as_uint(shaped_score(a, __uint_as_float(v[j]), r1h, r2h, rp - (base + j)));
            }
            bool waited = i == 0;                           // the weights' columns are free (the products of the tile before are done)
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
                const bool move = mx > m + (i == 0 ? 0.f : kTaLazy) || (m == -INFINITY && mx > -INFINITY);
                if (__any_sync(0xffffffffu, move)) {        // rare behind the first tiles: the reference of some row moves
                    const float f = move ? ex2(m - mx) : 1.f;
                    if (move) m = mx;
                    l *= f;                                 // (m = -inf: l is 0)
                    if (i > 0) {
                        if (!(ok = tc_spin_warp(o_full, (i - 1) & 1, quit))) break;
                        umb::tc_fence_after();
                        waited = true;
                        for (int c0 = 0; c0 < z.v_atoms * 64; c0 += 32) {
                            uint32_t o[32];
                            UMB_TMEM_LD_X32(t0 + 128 + c0, o);
                            umb::tc_wait_ld();
#pragma unroll
                            for (int j = 0; j < 32; ++j) o[j] = __float_as_uint(__uint_as_float(o[j]) * f);
                            UMB_TMEM_ST_X32(t0 + 128 + c0, o);
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
            // (asked in front of the parts, known behind them: a wait for a barrier that is through costs 200 to 350 clocks)
            const bool o_there = !waited && tc_test(o_full, (i - 1) & 1), s_there = i + 1 < kt.n && tc_test(s_full + ((i + 1) & 1), ((i + 1) >> 1) & 1);
            f32x2 l2[2] = {0ull, 0ull};
            uint32_t ph[16], pm[16];
#pragma unroll
            for (int j = 0; j < 16; ++j) {
                const float p = __uint_as_float(v[2 * j]), p1 = __uint_as_float(v[2 * j + 1]);
                const f32x2 pp = pack2(p, p1), r = add2(pp, pack2(minus_cut(p), minus_cut(p1)));
                const float2 ra = unpack2(r), rb = unpack2(add2(r, pack2(minus_cut(ra.x), minus_cut(ra.y))));
                l2[j & 1] = add2(l2[j & 1], pp);
                ph[j] = hi_pair(p, p1);
                pm[j] = hi_pair(ra.x, ra.y);
                v[j] = hi_pair(rb.x, rb.y);                                 // (v[2 j] and v[2 j + 1] have been used)
            }
            const float2 la = unpack2(l2[0]), lb = unpack2(l2[1]);
            l += (la.x + la.y) + (lb.x + lb.y);
            if (!waited) {
                if (!__all_sync(0xffffffffu, o_there) && !(ok = tc_spin_warp(o_full, (i - 1) & 1, quit))) break;
                umb::tc_fence_after();
            }
            s_ready = __all_sync(0xffffffffu, s_there);
            UMB_TMEM_ST_X16(t0 + 64, ph);
            UMB_TMEM_ST_X16(t0 + 80, pm);
            UMB_TMEM_ST_X16(t0 + 96, v);
            umb::tc_wait_st();
            umb::tc_fence_before();
            __syncwarp();
            if (lane == 0) umb::mbar_arrive(p_full);
        }
        if (ok) ok = tc_spin_warp(o_full, (kt.n - 1) & 1, quit);
        if (ok) {
            umb::tc_fence_after();
            const float inv = MODE == UMBS_ATTN_SIGMOID ? 1.f : 1.f / l;
            const int64_t t = start + r;
            const float* grow = a.gate ? a.gate + t * a.ldg + (a.gate_per_head ? h : h * a.vdim) : nullptr;
            const float gh = (grow && a.gate_per_head && r < len) ? sigmoidf_(grow[0]) : 1.f;
            const bool gvec = grow && !a.gate_per_head && ((uintptr_t)grow & 15) == 0;
            __nv_bfloat16* orow = STEP ? (__nv_bfloat16*)x.out + t * x.ldo + (int64_t)h * a.vdim
                                       : (__nv_bfloat16*)a.out + t * a.heads * a.vdim + (int64_t)h * a.vdim;
            float odd = 0.f;                                // stays 0 while the row's sums are finite
            for (int c0 = 0; c0 < a.vdim; c0 += 32) {
                uint32_t v[32];
                UMB_TMEM_LD_X32(t0 + 128 + c0, v);
                umb::tc_wait_ld();
                if (r < len) {
#pragma unroll
                    for (int e = 0; e < 32; e += 8) {
                        if (c0 + e < a.vdim) {                              // (vdim is a multiple of 8)
                            float o[8];
#pragma unroll
                            for (int u = 0; u < 8; ++u) {
                                o[u] = __uint_as_float(v[e + u]) * inv;
                                odd = fmaf(o[u], 0.f, odd);
                            }
                            if (grow) {
                                float g[8];
                                if (gvec) {
                                    *reinterpret_cast<float4*>(g) = *reinterpret_cast<const float4*>(grow + c0 + e);
                                    *reinterpret_cast<float4*>(g + 4) = *reinterpret_cast<const float4*>(grow + c0 + e + 4);
                                }
#pragma unroll
                                for (int u = 0; u < 8; ++u)
                                    o[u] *= a.gate_per_head ? gh : sigmoidf_(gvec ? g[u] : grow[c0 + e + u]);
                            }
                            uint32_t w[4];
#pragma unroll
                            for (int u = 0; u < 4; ++u) {
                                const __nv_bfloat162 pr = __floats2bfloat162_rn(o[2 * u], o[2 * u + 1]);
                                w[u] = *reinterpret_cast<const uint32_t*>(&pr);
                            }
                            *reinterpret_cast<uint4*>(orow + c0 + e) = make_uint4(w[0], w[1], w[2], w[3]);
                        }
                    }
                }
                __syncwarp();
            }
            for (uint32_t rows = __ballot_sync(0xffffffffu, odd != 0.f); rows != 0; rows &= rows - 1)
                plain_row<MODE, STEP>(a, x, b, s, vh, q0 + warp * 32 + __ffs(rows) - 1);
        }
    }
    __syncwarp();
    umb::tc_fence_before();
    __syncthreads();
    tc_settle(quit, z.report);
    if (warp == 4) {
        umb::tc_fence_after();
        umb::tmem_dealloc(tmem, 256);
    }
}

// As many key and value tiles as leave room for a second block on the SM (228 KB, 1 KB of it per block the system's): four, or
// three beside queries of more than 128 numbers.
constexpr int kTaTiles = 110 * 1024, kTaSmem = 1024 + kTaTiles;     // the largest of them
static TaDims ta_dims(const CachedAttnArgs& a) {
    TaDims z{(a.dim + 63) / 64, (a.dim + 15) / 16, (a.vdim + 63) / 64, kTaStages, 0, nullptr};
    while (z.stages > 3 && z.q_atoms * (kTaQ * 128) + z.stages * (z.q_atoms + z.v_atoms) * (kTaK * 128) > kTaTiles) --z.stages;
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

template <int MODE, bool SHAPED, bool STEP>
static int launch_ta(const CachedAttnArgs& a, const StepKeys& x, const Batch& b, cudaStream_t st) {
    TaDims z = ta_dims(a);
    int rc = give_up_word(&z.report);
    if (rc == 0) rc = give_up_status();
    if (rc != 0) return rc;
    // heads that are whole pieces of 64 numbers: the step's rows as tensor maps.  Rows that overlap (a row repeated among them)
    // and whatever else a map does not describe are copied row by row like the other sizes.
    CUtensorMap mk{}, ms{}, mv{};
    z.tma = a.dim % 64 == 0 && a.vdim % 64 == 0 && (!STEP || (x.kdim % 64 == 0 && x.ldk >= (int64_t)a.heads * x.kdim && x.ldv >= (int64_t)a.heads * a.vdim &&
                                                              (x.kdim == a.dim || x.ldks >= a.dim - x.kdim)));
    if (z.tma) {
        if (STEP) {
            rc = encode_map(&mk, x.k, (uint64_t)a.heads * x.kdim, b.n_tokens, 1, x.ldk, 0, kTaK);
            if (rc == 0 && x.kdim < a.dim) rc = encode_map(&ms, x.ks, a.dim - x.kdim, b.n_tokens, 1, x.ldks, 0, kTaK);
            if (rc == 0) rc = encode_map(&mv, x.v, (uint64_t)a.heads * a.vdim, b.n_tokens, 1, x.ldv, 0, kTaK);
        } else {
            const uint64_t row = (uint64_t)a.kv_heads * (a.dim + a.vdim);
            rc = encode_map(&mk, a.kv, row, b.n_tokens, 1, row, 0, kTaK);
            mv = mk;
        }
        z.tma = rc == 0;
    }
    const int smem = 1024 + (z.q_atoms * (kTaQ + z.stages * kTaK) + z.stages * z.v_atoms * kTaK) * 128;
    auto kernel = attention_tc_kernel<MODE, SHAPED, STEP>;
    // (always the same limit: another thread may be between setting it and its launch)
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kTaSmem);
    if (e != cudaSuccess) return (int)e;
    return chain_launch(kernel, dim3((b.max_seq_len + kTaQ - 1) / kTaQ, a.heads, b.n_seqs), kTaThreads, smem, st, mk, ms, mv, a, x, b, z);
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
