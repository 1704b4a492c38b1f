// Products of 32-bit operands with more than a few rows on the 5th-generation tensor cores: C = A W^T, fp32 in, fp32 out.
//
// An fp32 number times 2^24 (so that no part falls below bf16's smallest number) is the sum of three bf16 numbers, rounded to nearest one
// after the other (8 significant bits each, the parts behind the first signed): 2^24 a = a0 + a1 + a2, exactly.  Products of bf16 numbers
// are exact in the tensor core, so
//     2^48 a w = a0 w0 + (a0 w1 + a1 w0 + a1 w1 + a0 w2 + a2 w0) + terms below 2^-26 of it.
// The tensor core cuts its running sums off where an fp32 addition rounds, so no long chain runs through it: a0 w0 is summed over
// 128 of k at a time, in two accumulators in turn, and these sums are added in fp32 registers; the small terms, 2^-8 of the result, have
// an accumulator of their own.  Distance from float64 at K = 64 / 512 / 1024 / 4096: 0.7 / 1.3 / 1.3 / 1.7e-7, where one chain of fp32
// multiply-adds has 1.4 / 4.0 / 5.7 / 11e-7.
//
// A persistent block per SM walks tiles of 128 rows x BN columns.  Warps 8-15 fetch fp32 rows a k step ahead, split them and
// write the three parts of both operands in the 128-byte-swizzled image; warp 16 issues the 24 products of a step of 64 k, which the tensor
// core takes no faster than it works them off; warps 0-7 add up and store.  Tensor memory: two accumulators of a0 w0 and the small
// terms', 3 BN of 512 columns.
//
// Bound: the splitting: 9 rows of 8 numbers a thread and step, and a step's loads, which nothing covers (2.6 us a step of 64 k at
// BN = 160, of which the products take 1.2).  777 rows of 1024 to 3088 columns: 177 us on the multiply-add pipe (its own time 66), 49 here; 64 rows
// 50 -> 28.  What the first forms cost: products issued by a splitting warp 100 us, activations unrolled into the kernel 77.
#include <algorithm>
#include <math.h>

#include "seq_gemm_walk.cuh"

namespace umbs {

constexpr int kSpMaxN = 160, kSpStages = 2, kSpConv = 8, kSpSum = 8;
constexpr int kSpThreads = 32 * (kSpConv + kSpSum + 1);
constexpr int kSpSmem = 1024 + kSpStages * 3 * (kTcRows + kSpMaxN) * 128;
constexpr int kSpChunk = 2;                                 // k steps whose a0 w0 the tensor core sums

// Where row r of the activations starts, in 16-byte pieces.  Rows that are gathered or follow other groups' may lie 64 GB and more behind A: the
// sums are told to work those out in plain fp32.
constexpr uint32_t kNoRow = 0xffffffffu;
__device__ __forceinline__ uint32_t piece(const GemmArgs& a, int64_t r) {
    const int64_t p = (a.row_src ? a.row_src[r] : r) * a.lda >> 2;
    return p < kNoRow ? (uint32_t)p : kNoRow;
}

__device__ __forceinline__ bool odd_sum(float s) { return !(fabsf(s) <= 3.402823466e38f); }

// What 16 neighbouring sums of a row become, in place (DUAL: u the up half).  Sums that the parts do not give are worked out again in
// plain fp32: of rows that piece() does not reach, of operands that are not finite or beyond 2^103 (a part is infinite then, the next NaN),
// and sums beyond 2^79 (2^127 in the scale of the parts).  16 side by side, for which a row's numbers are fetched once: all of 4096 rows x
// 1024 -> 1600 columns 28 -> 6.3 ms.  Out of line: unrolled into the kernel, its 80 copies were fetched from memory by every block, 40 us of
// a 77 us product.  again: counts them, and their way through a long row.
template <bool DUAL>
__device__ __noinline__ void finish_chunk(const GemmArgs& a, int g, int64_t row, int n0, float* v, float* u, int* again) {
    const float* A = (const float*)a.A + (int64_t)g * a.a_goff + (int64_t)(a.row_src ? a.row_src[row] : row) * a.lda;
    const float* W = (const float*)a.W + (int64_t)g * a.w_gstride;
#pragma unroll 1
    for (int h = 0; h < (DUAL ? 2 : 1); ++h) {
        float* o = h ? u : v;
        uint32_t odd = 0;
#pragma unroll
        for (int j = 0; j < 16; ++j) odd |= (uint32_t)(n0 + j < a.N && odd_sum(o[j])) << j;
        if (odd == 0) continue;
        const float* w = W + (int64_t)(h ? a.N + n0 : n0) * a.ldw;
        float s[16] = {};
#pragma unroll 1
        for (int k = 0; k < a.K; k += 4) {                  // (K is a multiple of 4, rows start on 16 bytes)
            const float4 x = *reinterpret_cast<const float4*>(A + k);
            uint32_t left = 0;                              // sums that are not NaN yet: those stay so
#pragma unroll
            for (int j = 0; j < 16; ++j)
                if (odd >> j & 1) {
                    const float4 y = __ldg(reinterpret_cast<const float4*>(w + j * a.ldw + k));
                    s[j] = fmaf(x.w, y.w, fmaf(x.z, y.z, fmaf(x.y, y.y, fmaf(x.x, y.x, s[j]))));
                    left |= (uint32_t)(s[j] == s[j]) << j;
                }
            if (left == 0) break;
            if ((k & 4095) == 0) atomicAdd(again, 1);
        }
#pragma unroll
        for (int j = 0; j < 16; ++j) o[j] = odd >> j & 1 ? s[j] : o[j];
    }
#pragma unroll 1
    for (int j = 0; j < 16 && n0 + j < a.N; ++j) v[j] = finish<DUAL>(a, v[j], DUAL ? u[j] : 0.f, g, row, n0 + j);
}

// A warp's wait whose time is up.  When all sums of a tile are worked out again, at 0.4 ms for 1024 of k and 16 of them, the warps that wait for these are in
// time as long as the count goes on: a wait gives up when its time is up once more with none in between.  (In the loops themselves a
// microsecond of 49.)
__device__ __noinline__ bool wait_on(uint64_t* bar, uint32_t parity, volatile int* quit, volatile int* again) {
    for (int seen = -1;;) {
        const int now = __shfl_sync(0xffffffffu, *again, 0);
        if (now == seen || __any_sync(0xffffffffu, *quit)) return tc_give_up(quit);
        seen = now;
        if (__all_sync(0xffffffffu, tc_poll_for(bar, parity, quit))) return true;
    }
}

#define UMBS_TMEM_LD_X8(taddr, r)                                                                                        \
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"                                \
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]) : "r"(taddr))

template <bool DUAL>
__global__ void __launch_bounds__(kSpThreads, 1) gemm_split_kernel(const __grid_constant__ GemmArgs a, const __grid_constant__ TcArgs t, const int bn) {
    extern __shared__ unsigned char smem_raw[];
    __shared__ uint64_t bars[2 * kSpStages + 5];
    __shared__ uint32_t s_tmem;
    __shared__ int s_quit, s_again;
    unsigned char* smem = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint64_t *full = bars, *empty = bars + kSpStages, *main_full = bars + 2 * kSpStages, *main_empty = main_full + 2, *low_empty = main_empty + 2;
    volatile int* quit = &s_quit;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int a_part = kTcRows * 128, w_part = bn * 128, stage = 3 * (a_part + w_part), out = DUAL ? bn / 2 : bn;
    if (threadIdx.x == 0) {
        for (int i = 0; i < kSpStages; ++i) {
            umb::mbar_init(full + i, kSpConv);
            umb::mbar_init(empty + i, 1);
        }
        for (int i = 0; i < 2; ++i) {
            umb::mbar_init(main_full + i, 1);
            umb::mbar_init(main_empty + i, kSpSum);
        }
        umb::mbar_init(low_empty, kSpSum);
        s_quit = s_again = 0;
        umb::fence_barrier_init();
    }
    if (warp == kSpConv + kSpSum) {
        umb::tmem_alloc(&s_tmem, 512);
        umb::tmem_relinquish();
    }
    umb::tc_fence_before();
    __syncthreads();
    umb::tc_fence_after();
    const uint32_t tmem = s_tmem;
    TileWalk w(a, t);
    auto poll = [&](uint64_t* bar, uint32_t parity) {
        return __all_sync(0xffffffffu, tc_poll_for(bar, parity, quit)) || wait_on(bar, parity, quit, &s_again);
    };
    auto spin = [&](uint64_t* bar, uint32_t parity) { return tc_spin_for(bar, parity) || wait_on(bar, parity, quit, &s_again); };

    if (warp < kSpSum) {
        // ------------------------------------------------------------------------------------ sums: a thread per row and half the columns
        const int q = warp & 3, half = warp >> 2, nch = bn / 32;           // chunks of 16 columns of this warp, at most five
        const uint32_t t0 = tmem + ((uint32_t)(q * 32) << 16);
        auto col = [&](int c) {                                            // (DUAL: the gate chunks, then their up chunks)
            return DUAL ? (c < nch / 2 ? half * (nch / 2) + c : nch + half * (nch / 2) + c - nch / 2) * 16 : (half * nch + c) * 16;
        };
        uint32_t it = 0;                                                   // chunks of k behind
        bool ok = true;
        while (ok && w.step()) {
            float acc[kSpMaxN / 32][16];
            auto add = [&](uint32_t at) {
#pragma unroll
                for (int c = 0; c < kSpMaxN / 32; ++c)
                    if (c < nch)
#pragma unroll
                        for (int h = 0; h < 16; h += 8) {
                            uint32_t v[8];
                            UMBS_TMEM_LD_X8(t0 + at + col(c) + h, v);
                            umb::tc_wait_ld();
#pragma unroll
                            for (int j = 0; j < 8; ++j) acc[c][h + j] += __uint_as_float(v[j]);
                        }
                umb::tc_fence_before();
                __syncwarp();
            };
#pragma unroll
            for (int c = 0; c < kSpMaxN / 32; ++c)
#pragma unroll
                for (int j = 0; j < 16; ++j) acc[c][j] = 0.f;
            for (int k = 0; ok && k < t.k_steps; k += kSpChunk, ++it) {
                const uint32_t m = it & 1;
                if (!(ok = poll(main_full + m, (it >> 1) & 1))) break;
                umb::tc_fence_after();
                add(m * bn);
                if (lane == 0) umb::mbar_arrive(main_empty + m);
            }
            if (!ok) break;
            add(2 * bn);                                                   // (the last chunk's barrier stands behind the small terms too)
            if (lane == 0) umb::mbar_arrive(low_empty);
#pragma unroll
            for (int c = 0; c < kSpMaxN / 32; ++c)
#pragma unroll
                for (int j = 0; j < 16; ++j) acc[c][j] *= kSplitBack;
            const int r = w.m0 + q * 32 + lane;
            if (r < w.rows && piece(a, w.row_lo + r) == kNoRow) {          // (nothing was summed for it)
#pragma unroll
                for (int c = 0; c < kSpMaxN / 32; ++c)
#pragma unroll
                    for (int j = 0; j < 16; ++j) acc[c][j] = NAN;
            }
            if (r < w.rows) {
                const int64_t grow = w.row_lo + r;
                float* crow = (float*)a.C + (int64_t)w.g * a.c_goff + grow * a.ldc;
#pragma unroll
                for (int c = 0; c < (DUAL ? kSpMaxN / 64 : kSpMaxN / 32); ++c) {
                    if (c >= (DUAL ? nch / 2 : nch)) continue;
                    const int n0 = w.n0 * out + col(c);
                    bool odd = DUAL || a.bias != nullptr || a.unary != 0 || a.out_gate != nullptr;
#pragma unroll
                    for (int j = 0; j < 16; ++j) odd |= odd_sum(acc[c][j]);
                    if (odd) {
                        float o[16], up[16];
#pragma unroll
                        for (int j = 0; j < 16; ++j) {
                            o[j] = acc[c][j];
                            if (DUAL) up[j] = nch == 4 ? acc[c + 2][j] : acc[c + 1][j];
                        }
                        finish_chunk<DUAL>(a, w.g, grow, n0, o, up, &s_again);
#pragma unroll
                        for (int j = 0; j < 16; ++j) acc[c][j] = o[j];
                    }
                    const float* o = acc[c];
#pragma unroll
                    for (int j = 0; j < 16; j += 4) {
                        if (t.vec_c && n0 + j + 4 <= a.N) *reinterpret_cast<float4*>(crow + n0 + j) = make_float4(o[j], o[j + 1], o[j + 2], o[j + 3]);
                        else
#pragma unroll
                            for (int e = 0; e < 4; ++e)
                                if (n0 + j + e < a.N) crow[n0 + j + e] = o[j + e];
                    }
                }
            }
            __syncwarp();
        }
    } else if (warp < kSpSum + kSpConv) {
        // ------------------------------------------------------------------------------------ operands: eight threads per row of 64 k
        constexpr int kRows = kSpConv * 4, PA = kTcRows / kRows, PW = kSpMaxN / kRows, P = PA + PW;     // rows side by side; rows of a thread
        const int tid = threadIdx.x - kSpSum * 32, ch = tid & 7, r0 = tid >> 3, pw = bn / kRows;
        const uint32_t base = smem_u32(smem) + r0 * 128 + ((ch ^ (r0 & 7)) << 4);
        uint32_t it = 0;
        bool ok = true;
        while (ok && w.step()) {
            const float4* A = (const float4*)((const float*)a.A + (int64_t)w.g * a.a_goff) + ch * 2;
            const float4* W = (const float4*)((const float*)a.W + (int64_t)w.g * a.w_gstride) + ch * 2;
            uint32_t off[P];                                               // where a row starts, in 16-byte pieces; kNoRow: none here, zeros
#pragma unroll
            for (int p = 0; p < PA; ++p) {
                const int r = w.m0 + p * kRows + r0;
                off[p] = r < w.rows ? piece(a, w.row_lo + r) : kNoRow;
            }
#pragma unroll
            for (int p = 0; p < PW; ++p) {
                const int r = p * kRows + r0, n = w.n0 * out + (DUAL && r >= out ? r - out : r);
                off[PA + p] = p < pw && n < a.N ? (uint32_t)((int64_t)(DUAL && r >= out ? a.N + n : n) * a.ldw >> 2) : kNoRow;
            }
            float4 buf[P][2];
            auto fetch = [&](int k) {
                const int left = a.K - k * kTcK - ch * 8;                  // (K is a multiple of 4; behind the last step: nothing)
#pragma unroll
                for (int p = 0; p < P; ++p)
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        buf[p][e] = make_float4(0.f, 0.f, 0.f, 0.f);
                        if (off[p] != kNoRow && left > 4 * e) buf[p][e] = (p < PA ? A : W)[(uint64_t)off[p] + k * (kTcK / 4) + e];
                    }
            };
            fetch(0);
            for (int k = 0; k < t.k_steps; ++k, ++it) {
                const uint32_t s = it % kSpStages;
                if (!(ok = poll(empty + s, ((it / kSpStages) & 1) ^ 1))) break;
                const uint32_t dst = base + s * stage;
#pragma unroll
                for (int p = 0; p < P; ++p) {
                    if (p < PA + pw) {
                        const float f[8] = {buf[p][0].x, buf[p][0].y, buf[p][0].z, buf[p][0].w, buf[p][1].x, buf[p][1].y, buf[p][1].z, buf[p][1].w};
                        uint4 v[3];
                        split8(f, v);
                        const uint32_t d = dst + (p < PA ? p * kRows * 128 : 3 * a_part + (p - PA) * kRows * 128), step = p < PA ? a_part : w_part;
#pragma unroll
                        for (int e = 0; e < 3; ++e)
                            asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(d + e * step), "r"(v[e].x), "r"(v[e].y), "r"(v[e].z), "r"(v[e].w) : "memory");
                    }
                }
                umb::fence_proxy_async_smem();
                __syncwarp();
                if (lane == 0) umb::mbar_arrive(full + s);
                // behind the fence, which waits for a thread's loads too, and all at once: a load that is waited for is waited for together with
                // those asked for behind it (each row where the one before it has been split: 66 us instead of 48)
                fetch(k + 1);
            }
        }
    } else {
        // ------------------------------------------------------------------------------------ products
        const uint32_t idesc = tc_idesc(kTcRows, bn), d_low = tmem + 2 * bn;
        uint32_t it = 0, chunk = 0, tiles = 0;
        bool ok = true;
        for (; ok && w.step(); ++tiles) {
            if (!(ok = spin(low_empty, (tiles & 1) ^ 1))) break;
            for (int k = 0; k < t.k_steps; ++k, ++it) {
                const uint32_t s = it % kSpStages, m = chunk & 1;
                if (k % kSpChunk == 0 && !(ok = spin(main_empty + m, ((chunk >> 1) & 1) ^ 1))) break;
                if (!(ok = spin(full + s, (it / kSpStages) & 1))) break;
                umb::tc_fence_after();
                const uint32_t st = smem_u32(smem) + s * stage, d_main = tmem + m * bn, go_main = k % kSpChunk ? 1u : 0u, go_low = k ? 1u : 0u;
                const bool last = k + 1 == t.k_steps || k % kSpChunk == kSpChunk - 1;
                const uint64_t ad = umb::umma_smem_desc_sw128(st), wd = umb::umma_smem_desc_sw128(st + 3 * a_part);
                if (umb::elect_one()) {
#pragma unroll
                    for (int kk = 0; kk < kTcK / 16; ++kk)
#pragma unroll
                        for (int i = 0; i < 3; ++i)
#pragma unroll
                            for (int j = 0; j < 3 - i; ++j)
                                umb::umma_ss_f16(i + j ? d_low : d_main, ad + i * (a_part >> 4) + kk * 2, wd + j * (w_part >> 4) + kk * 2, idesc,
                                                 kk > 0 || i + j > 1 || i > 0 ? 1u : (i + j ? go_low : go_main));
                    umb::umma_commit(empty + s);
                    if (last) umb::umma_commit(main_full + m);
                }
                __syncwarp();
                if (last) ++chunk;
            }
        }
    }
    __syncwarp();
    umb::tc_fence_before();
    __syncthreads();
    tc_settle(quit, t.report);
    if (warp == kSpConv + kSpSum) {
        umb::tc_fence_after();
        umb::tmem_dealloc(tmem, 512);
    }
}

int launch_gemm_split(const GemmArgs& a, int groups, bool dual, cudaStream_t st) {
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
    t.k_steps = (a.K + kTcK - 1) / kTcK;
    t.vec_c = (uintptr_t)a.C % 16 == 0 && a.ldc % 4 == 0 && a.c_goff % 4 == 0;
    const int64_t m = a.grp_off != nullptr ? (int64_t)groups * ((a.M + groups * kTcRows - 1) / (groups * kTcRows)) : (int64_t)groups * t.m_tiles;
    int bn = 0;
    int64_t best = 0;
    for (int c = dual ? 64 : 32; c <= (dual ? 128 : kSpMaxN); c += dual ? 64 : 32) {
        const int o = dual ? c / 2 : c;
        // rounds of tiles over the SMs times a step's length (measured: 1.2 us at 32 columns, 2.6 at 160)
        const int64_t cost = (m * ((a.N + o - 1) / o) + sms - 1) / sms * (85 + 11 * (c / 10));
        if (bn == 0 || cost < best) {
            bn = c;
            best = cost;
        }
    }
    const int o = dual ? bn / 2 : bn;
    t.n_tiles = (a.N + o - 1) / o;
    const int64_t tiles = (int64_t)t.groups * t.m_tiles * t.n_tiles;            // (sorted by expert: at most)
    auto run = [&](auto kernel) -> int {
        const cudaError_t er = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSpSmem);
        if (er != cudaSuccess) return (int)er;
        kernel<<<(int)(tiles < sms ? tiles : sms), kSpThreads, kSpSmem, st>>>(a, t, bn);
        return 0;
    };
    return dual ? run(gemm_split_kernel<true>) : run(gemm_split_kernel<false>);
}

unsigned int split_timeouts() { return tc_timeouts(); }

}  // namespace umbs
