// The output tiles of a persistent block of the tensor-core products (seq_gemm_tc.cu, seq_gemm_split.cu).
#pragma once
#include "seq_gemm.h"
#include "seq_tc.cuh"

namespace umbs {

constexpr int kTcRows = 128, kTcK = 64;                     // tile rows; k per ring stage

struct TcArgs {
    int groups, n_tiles, m_tiles, k_steps;
    int vec_c;                                              // rows of C take 16-byte (fp32) / 8-byte (bf16) stores of 4 columns
    int a_grouped, w_grouped;                               // the group coordinate of the tensor maps is used
    unsigned int* report;                                   // give_up_word()
};

// The tiles of a block, in the order every role visits them: rows fastest, then columns, then groups.
struct TileWalk {
    const GemmArgs& a; const TcArgs& t;
    int next, g, first, m_tiles, row_lo, rows, m0, n0;
    __device__ TileWalk(const GemmArgs& a_, const TcArgs& t_) : a(a_), t(t_), next(blockIdx.x), g(-1), first(0), m_tiles(0), row_lo(0), rows(a_.M), m0(0), n0(0) {}
    __device__ bool step() {
        while (next >= first + m_tiles * t.n_tiles) {
            if (++g >= t.groups) return false;
            first += m_tiles * t.n_tiles;
            if (a.grp_off != nullptr) {
                row_lo = a.grp_off[g];
                rows = a.grp_off[g + 1] - row_lo;
                m_tiles = (rows + kTcRows - 1) / kTcRows;
            } else {
                m_tiles = t.m_tiles;
            }
        }
        const int i = next - first;
        m0 = i % m_tiles * kTcRows;
        n0 = i / m_tiles;                                   // in tiles: the caller knows their width
        next += gridDim.x;
        return true;
    }
};

constexpr int kTcStageRow = 36;                             // fp32 row stride of an epilogue warp's 32 x 32 staging block (32 x 16: 20)

// Bias and activation of C neighbouring columns of a row, v (and u, the up half) in place.  One choice of activation in
// front of a loop over independent elements: chosen element by element, every exponential and every quotient waited for the
// one before it (25 to 40 us for a tile's 128 x 128 outputs, several times its products).
template <bool DUAL, int C>
__device__ __forceinline__ void tc_finish(const GemmArgs& a, uint32_t (&v)[C], uint32_t (&u)[DUAL ? C : 1], int n0) {
#define UMBS_F(x) __uint_as_float(x)
#define UMBS_EACH(expr)                                                                     \
    _Pragma("unroll") for (int j = 0; j < C; ++j) {                                        \
        const float x = UMBS_F(v[j]), y = DUAL ? UMBS_F(u[DUAL ? j : 0]) : 0.f;              \
        v[j] = __float_as_uint(expr);                                                       \
        (void)y;                                                                            \
    }
    if (a.bias != nullptr) {
#pragma unroll
        for (int j = 0; j < C; ++j) {
            const int n = min(n0 + j, a.N - 1);
            v[j] = __float_as_uint(UMBS_F(v[j]) + a.bias[n]);
            if (DUAL) u[DUAL ? j : 0] = __float_as_uint(UMBS_F(u[DUAL ? j : 0]) + a.bias[a.N + n]);
        }
    }
    if (DUAL) {
        if (a.act == UMBS_ACT_GELU_TANH) UMBS_EACH(gated_act(x, y, a.limit, UMBS_ACT_GELU_TANH))
        else if (a.act == UMBS_ACT_SILU) UMBS_EACH(x * tc_sigmoid(x) * y)
        else UMBS_EACH(fminf(x, a.limit) * tc_sigmoid(1.702f * fminf(x, a.limit)) * (fminf(fmaxf(y, -a.limit), a.limit) + 1.f))
    } else if (a.unary && n0 + C <= a.unary_cols && (a.unary == UMBS_UNARY_SILU || a.unary == UMBS_UNARY_RELU2 || a.unary == UMBS_UNARY_SCALE)) {
        if (a.unary == UMBS_UNARY_SILU) UMBS_EACH(x * tc_sigmoid(x))
        else if (a.unary == UMBS_UNARY_RELU2) UMBS_EACH(unary_act(x, UMBS_UNARY_RELU2, a.p0, a.p1))
        else UMBS_EACH(unary_act(x, UMBS_UNARY_SCALE, a.p0, a.p1))
    } else if (a.unary) {
        UMBS_EACH(n0 + j < a.unary_cols ? unary_act(x, a.unary, a.p0, a.p1) : x)
    }
#undef UMBS_EACH
#undef UMBS_F
}

template <int C> __device__ __forceinline__ void tc_load(uint32_t addr, uint32_t (&v)[C]) {
    if constexpr (C == 32) UMB_TMEM_LD_X32(addr, v);
    else UMB_TMEM_LD_X16(addr, v);
}
// 32 rows of a finished tile, by a warp: kOut columns from tensor memory `src` (DUAL: the gate columns, the up columns kUp behind them) through
// its staging block, CW columns at a time, to rows grow .. of C, of which `rows` are there, from column col on.  read_done: by one lane once tensor
// memory is read.
template <int kOut, int kUp, bool DUAL, typename TC, int CW = 32, typename F>
__device__ __forceinline__ void tc_store_tile(const GemmArgs& a, int vec_c, uint32_t src, float* so, int g, int64_t grow, int rows, int col, F&& read_done) {
    constexpr int kRow = CW + 4, kLanes = CW / 4, kRows = 32 / kLanes;      // staging row; lanes of a row piece; rows side by side
    const int lane = threadIdx.x & 31, rr = lane / kLanes, cc = lane % kLanes * 4, n_hi = a.N - col;
    TC* C = (TC*)a.C + (int64_t)g * a.c_goff + grow * a.ldc + col;
#pragma unroll 1
    for (int c0 = 0; c0 < kOut; c0 += CW) {
        uint32_t v[CW], u[DUAL ? CW : 1];
        tc_load(src + c0, v);
        if constexpr (DUAL) tc_load(src + kUp + c0, u);
        umb::tc_wait_ld();
        if (c0 + CW >= kOut) {                              // read to the end: the next tile but one may be summed here
            umb::tc_fence_before();
            __syncwarp();
            if (lane == 0) read_done();
        }
        if (c0 >= n_hi || rows <= 0) continue;
        if (DUAL || a.bias != nullptr || a.unary) tc_finish<DUAL, CW>(a, v, u, col + c0);
#pragma unroll
        for (int j = 0; j < CW; j += 4) *reinterpret_cast<uint4*>(so + lane * kRow + j) = make_uint4(v[j], v[j + 1], v[j + 2], v[j + 3]);
        __syncwarp();
#pragma unroll
        for (int i = 0; i < 32 / kRows; ++i) {
            const int r = i * kRows + rr, n = c0 + cc;
            if (r < rows && n < n_hi) {
                const float4 f = *reinterpret_cast<const float4*>(so + r * kRow + cc);
                float o[4] = {f.x, f.y, f.z, f.w};
                if (a.out_gate != nullptr) {
#pragma unroll
                    for (int e = 0; e < 4; ++e)
                        if (n + e < n_hi) o[e] = finish_gate(a, o[e], g, grow + r, col + n + e);
                }
                TC* p = C + (int64_t)r * a.ldc + n;
                if (vec_c && n + 4 <= n_hi) {
                    if constexpr (sizeof(TC) == 4) {
                        *reinterpret_cast<float4*>(p) = make_float4(o[0], o[1], o[2], o[3]);
                    } else {
                        __nv_bfloat162 lo = __floats2bfloat162_rn(o[0], o[1]), hi = __floats2bfloat162_rn(o[2], o[3]);
                        *reinterpret_cast<uint2*>(p) = make_uint2(*reinterpret_cast<uint32_t*>(&lo), *reinterpret_cast<uint32_t*>(&hi));
                    }
                } else {
#pragma unroll
                    for (int e = 0; e < 4; ++e)
                        if (n + e < n_hi) p[e] = from_f32<TC>(o[e]);
                }
            }
        }
        __syncwarp();
    }
}

// seq_gemm_pair.cu: dense rows, tiles of 256 rows by pairs of SMs
int launch_gemm_pair(const GemmArgs& a, TcArgs t, bool dual, bool c_f32, int sms, cudaStream_t st);

}  // namespace umbs
