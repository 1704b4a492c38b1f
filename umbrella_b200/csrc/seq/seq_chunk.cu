// Matrix memories whose decay is one number per head and token, for steps with many tokens: instead of walking the tokens one by
// one, 32 of them are a few products of small matrices.  With D[i][j] the product of the decays behind token j up to token i
// times j's weight (0 for j > i), and L[i] the product of the decays up to i,
//     O = diag(L) Q S + ((Q K^T) o D) V,        S <- L[last] S + (diag(D[last]) K)^T V.
// Same sums as the walk up to the order of additions, fp32 throughout (two products per instruction).
//
// One block = (sequence or segment of it, head, 128 value columns), 256 threads, two blocks on an SM; the state and the 32
// tokens' rows sit in shared memory, the next tokens' rows are on their way in registers.  A thread of Q S and of D V owns four
// rows x four columns, of K^T V four rows x eight columns: two or three 16-byte loads for 16 or 32 multiply-adds.
// Walking tokens: a token's state update is a chain of shared-memory loads that every warp of a block repeats, 0.1 us per token
// and block; 4096 tokens, 16 heads of 64 x 128 took 822 us in its two passes, these 194 us
// (retention of that size is seq_chunk_tc.cu's now: 119 with norm and gate).
#include <algorithm>
#include <math.h>

#include "seq_chunk.h"

namespace umbs {

constexpr int kChD = 64, kChV = 128;                       // largest key size; value columns of a block
constexpr int kChT = kChunkTokens, kChQ = kChT + 4, kChK = kChD + 4, kChS = kChV + 4;      // padded row lengths

struct ChunkShared {
    float q[kChD][kChQ], k[kChD][kChQ];                    // [dimension][token]
    float kw[kChT][kChK];                                  // [token][dimension], times the weight the token keeps to the end
    float v[kChT][kChS];                                   // [token][column]
    float p[kChT][kChQ];                                   // [key token][query token]: D, then (Q K^T) o D
    float s[kChD][kChS];                                   // the state
    float n[kChD];                                         // its normaliser column
    float a[kChT], bw[kChT], lam[kChT], keep[kChT];        // decays, weights, L, D[last]
};

__device__ __forceinline__ ulonglong2 ld2(const float* p) { return *reinterpret_cast<const ulonglong2*>(p); }

template <bool GATES>
__global__ void __launch_bounds__(256, 2) chunk_memory_kernel(const ChunkMemory x, const Batch b) {
    extern __shared__ __align__(16) unsigned char smem[];
    ChunkShared& sh = *reinterpret_cast<ChunkShared*>(smem);
    chain_wait();
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int s = blockIdx.x / x.n_seg, seg = blockIdx.x - s * x.n_seg, h = blockIdx.y, c0 = blockIdx.z * kChV;
    const int seq_len = b.seq_len[s], t_first = seg * x.seg_len;
    if (t_first >= seq_len) return;
    const int len = min(x.seg_len, seq_len - t_first), start = b.seq_start[s] + t_first;
    const bool last_seg = t_first + len == seq_len, cut = x.pass != 0;
    if (x.pass == 1 && last_seg) return;
    const int dim = x.dim, vdim = x.vdim, nv = min(kChV, vdim - c0), V1 = vdim + x.normaliser;
    const bool norm = GATES && x.normaliser && c0 == 0;     // this block carries the normaliser
    const int64_t plane = (int64_t)x.heads * dim * V1;
    float* st = x.state + ((int64_t)b.seq_slot[s] * x.heads + h) * x.state_stride;
    const float* st_in = b.seq_pos0[s] > 0 && x.pass != 1 ? st : nullptr;
    if (x.pass == 2 && !(seg == 0 && last_seg))             // (segment 0 of a cut sequence: the chain kernel's copy of the slot's state)
        st_in = x.seg_state + ((int64_t)s * x.n_seg + (seg > 0 ? seg - 1 : x.n_seg - 1)) * plane + (int64_t)h * dim * V1;
    for (int i = tid; i < kChD * kChV; i += 256) {
        const int d = i / kChV, c = i - d * kChV;
        sh.s[d][c] = st_in != nullptr && d < dim && c < nv ? st_in[(int64_t)d * V1 + c0 + c] : 0.f;
    }
    if (tid < kChD) sh.n[tid] = norm && st_in != nullptr && tid < dim ? st_in[(int64_t)tid * V1 + vdim] : 0.f;
    const float dec = GATES ? 0.f : x.decay[h];
    if (!GATES && tid < kChT) sh.lam[tid] = powf(dec, (float)(tid + 1));
    float total = 1.f;                                      // product of the segment's decays
    const int half = x.rot_dims / 2;

    // rows of the 32 tokens from t0: q and k 8 numbers a thread (lane: dimension), v 16 (lane: column), the turn's cos and sin
    float pq[8], pk[8], pv[16], pc[4], ps[4], pa = 1.f, pb = 0.f;
    auto fetch = [&](int t0) {
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            const int i = warp * 4 + (e >> 1), d = (e & 1) * 32 + lane;
            const bool ok = t0 + i < len && d < dim;
            const float* row = x.x + (int64_t)(start + t0 + i) * x.ld;
            pq[e] = ok ? row[x.qoff + h * dim + d] * x.qscale : 0.f;
            pk[e] = ok ? row[x.koff + h * dim + d] * x.kscale : 0.f;
        }
#pragma unroll
        for (int e = 0; e < 16; ++e) {
            const int i = warp * 4 + (e >> 2), c = (e & 3) * 32 + lane;
            pv[e] = t0 + i < len && c < nv ? x.x[(int64_t)(start + t0 + i) * x.ld + x.voff + h * vdim + c0 + c] : 0.f;
        }
        if (x.rot_dims > 0) {
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int i = warp * 4 + e;
                const bool ok = t0 + i < len && lane < half;
                const float* row = x.rot_tab + (int64_t)(start + t0 + i) * x.rot_dims;
                pc[e] = ok ? row[lane] : 1.f;
                ps[e] = ok ? row[half + lane] : 0.f;
            }
        }
        if (GATES && tid < kChT) {
            const bool ok = t0 + tid < len;
            const float* g = x.gates + ((int64_t)(start + t0 + tid) * x.heads + h) * 3;
            pa = ok ? g[0] : 1.f;
            pb = ok ? g[1] : 0.f;
        }
    };
    fetch(0);
    for (int t0 = 0; t0 < len; t0 += kChT) {
        const int nb = min(kChT, len - t0);
        __syncthreads();                                    // the tokens before are done with
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            const int i = warp * 4 + (e >> 1), d = (e & 1) * 32 + lane;
            sh.q[d][i] = pq[e];
            sh.k[d][i] = pk[e];
        }
#pragma unroll
        for (int e = 0; e < 16; ++e) sh.v[warp * 4 + (e >> 2)][(e & 3) * 32 + lane] = pv[e];
        if (GATES && tid < kChT) {
            sh.a[tid] = pa;
            sh.bw[tid] = pb;
        }
        if (!GATES && tid < kChT) sh.keep[tid] = tid >= nb ? 0.f : (tid == nb - 1 ? 1.f : sh.lam[nb - 2 - tid]);
        if (x.rot_dims > 0) {
            __syncwarp();                                   // a warp turns the four tokens it wrote: (u, v) -> (u cos - v sin, v cos + u sin)
            if (lane < half)
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int i = warp * 4 + e;
                    const float qu = sh.q[lane][i], qv = sh.q[lane + half][i], ku = sh.k[lane][i], kv = sh.k[lane + half][i];
                    sh.q[lane][i] = qu * pc[e] - qv * ps[e];
                    sh.q[lane + half][i] = qv * pc[e] + qu * ps[e];
                    sh.k[lane][i] = ku * pc[e] - kv * ps[e];
                    sh.k[lane + half][i] = kv * pc[e] + ku * ps[e];
                }
        }
        __syncthreads();
        if (GATES && warp == 0) {                           // lane j: column j of D, one decay after the other
            float dj = sh.bw[lane], lam = 1.f;
            for (int i = 0; i < kChT; ++i) {
                const float ai = sh.a[i];
                lam *= ai;
                if (i > lane) dj *= ai;
                sh.p[lane][i] = i >= lane ? dj : 0.f;
                if (lane == 0) sh.lam[i] = lam;
            }
            sh.keep[lane] = dj;                             // (decays behind the last token are 1)
            total *= lam;
        }
        if (t0 + kChT < len) fetch(t0 + kChT);
        if (GATES) __syncthreads();
        // keys as they will be kept, token by token
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            const int d = warp * 8 + e;
            sh.kw[lane][d] = sh.k[d][lane] * sh.keep[lane];
        }
        if (x.pass != 1) {
            const int ti = (tid >> 4) * 2, tj = (tid & 15) * 2;             // (Q K^T) o D: two query tokens x two key tokens
            float acc[2][2] = {};
            if (tj <= ti + 1) {
#pragma unroll 8
                for (int d = 0; d < dim; ++d) {
                    const float2 qv = *reinterpret_cast<const float2*>(&sh.q[d][ti]), kv = *reinterpret_cast<const float2*>(&sh.k[d][tj]);
                    acc[0][0] = fmaf(qv.x, kv.x, acc[0][0]);
                    acc[0][1] = fmaf(qv.x, kv.y, acc[0][1]);
                    acc[1][0] = fmaf(qv.y, kv.x, acc[1][0]);
                    acc[1][1] = fmaf(qv.y, kv.y, acc[1][1]);
                }
            }
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    const int far = ti + i - (tj + j);
                    const float f = GATES ? sh.p[tj + j][ti + i] : (far <= 0 ? 1.f : sh.lam[far - 1]);
                    sh.p[tj + j][ti + i] = far < 0 ? 0.f : acc[i][j] * f;   // (chosen, not multiplied by 0: a later token's NaN stays its own)
                }
        }
        __syncthreads();
        if (x.pass != 1) {
            const int i0 = warp * 4, c = lane * 4;
            if (i0 < nb) {
                f32x2 acc[4][2] = {};
#pragma unroll 4
                for (int d = 0; d < dim; ++d) {
                    const float4 qv = *reinterpret_cast<const float4*>(&sh.q[d][i0]);
                    const ulonglong2 sv = ld2(&sh.s[d][c]);
                    const float qa[4] = {qv.x, qv.y, qv.z, qv.w};
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const f32x2 qq = pack2(qa[i], qa[i]);
                        acc[i][0] = fma2(qq, sv.x, acc[i][0]);
                        acc[i][1] = fma2(qq, sv.y, acc[i][1]);
                    }
                }
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float f = sh.lam[i0 + i];
                    acc[i][0] = mul2(acc[i][0], pack2(f, f));
                    acc[i][1] = mul2(acc[i][1], pack2(f, f));
                }
#pragma unroll 4
                for (int j = 0; j < i0; ++j) {                          // tokens that all four rows see
                    const float4 pv4 = *reinterpret_cast<const float4*>(&sh.p[j][i0]);
                    const ulonglong2 vv = ld2(&sh.v[j][c]);
                    const float pp[4] = {pv4.x, pv4.y, pv4.z, pv4.w};
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const f32x2 q2 = pack2(pp[i], pp[i]);
                        acc[i][0] = fma2(q2, vv.x, acc[i][0]);
                        acc[i][1] = fma2(q2, vv.y, acc[i][1]);
                    }
                }
#pragma unroll
                for (int e = 0; e < 4; ++e) {                           // the rows' own tokens: seen by themselves and the rows behind
                    if (i0 + e >= nb) break;
                    const ulonglong2 vv = ld2(&sh.v[i0 + e][c]);
#pragma unroll
                    for (int i = e; i < 4; ++i) {
                        const float w = sh.p[i0 + e][i0 + i];
                        const f32x2 q2 = pack2(w, w);
                        acc[i][0] = fma2(q2, vv.x, acc[i][0]);
                        acc[i][1] = fma2(q2, vv.y, acc[i][1]);
                    }
                }
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    if (i0 + i >= nb || c >= nv) continue;
                    float* o = x.out + ((int64_t)(start + t0 + i0 + i) * x.heads + h) * V1 + c0 + c;
                    const float2 u = unpack2(acc[i][0]), w = unpack2(acc[i][1]);
                    if (!GATES && ((uintptr_t)o & 15) == 0) {               // (vdim is a multiple of four)
                        *reinterpret_cast<float4*>(o) = make_float4(u.x, u.y, w.x, w.y);
                    } else {
                        o[0] = u.x; o[1] = u.y; o[2] = w.x; o[3] = w.y;
                    }
                }
            }
            if (norm) {                                     // n . q: eight lanes per token
                const int i = tid >> 3, part = tid & 7;
                float z = 0.f, zp = 0.f;
                for (int d = part; d < dim; d += 8) z = fmaf(sh.q[d][i], sh.n[d], z);
                for (int j = part; j <= i; j += 8) zp += sh.p[j][i];
                z = fmaf(z, sh.lam[i], zp);
#pragma unroll
                for (int o = 4; o > 0; o >>= 1) z += __shfl_xor_sync(0xffffffffu, z, o);
                if (part == 0 && i < nb) x.out[((int64_t)(start + t0 + i) * x.heads + h) * V1 + vdim] = z;
            }
        }
        __syncthreads();                                    // the state in front of these tokens has been read
        const float kept = sh.lam[GATES ? kChT - 1 : nb - 1];
        {
            const int d = (tid >> 4) * 4, c = (tid & 15) * 4;
            f32x2 acc[4][4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const ulonglong2 s0 = ld2(&sh.s[d + i][c]), s1 = ld2(&sh.s[d + i][c + 64]);
                const f32x2 kk = pack2(kept, kept);
                acc[i][0] = mul2(s0.x, kk); acc[i][1] = mul2(s0.y, kk);
                acc[i][2] = mul2(s1.x, kk); acc[i][3] = mul2(s1.y, kk);
            }
#pragma unroll 4
            for (int j = 0; j < nb; ++j) {
                const float4 kv = *reinterpret_cast<const float4*>(&sh.kw[j][d]);
                const ulonglong2 v0 = ld2(&sh.v[j][c]), v1 = ld2(&sh.v[j][c + 64]);
                const float ka[4] = {kv.x, kv.y, kv.z, kv.w};
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const f32x2 kk = pack2(ka[i], ka[i]);
                    acc[i][0] = fma2(kk, v0.x, acc[i][0]);
                    acc[i][1] = fma2(kk, v0.y, acc[i][1]);
                    acc[i][2] = fma2(kk, v1.x, acc[i][2]);
                    acc[i][3] = fma2(kk, v1.y, acc[i][3]);
                }
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                *reinterpret_cast<ulonglong2*>(&sh.s[d + i][c]) = make_ulonglong2(acc[i][0], acc[i][1]);
                *reinterpret_cast<ulonglong2*>(&sh.s[d + i][c + 64]) = make_ulonglong2(acc[i][2], acc[i][3]);
            }
            if (norm && tid < kChD) {
                float z = sh.n[tid] * kept;
                for (int j = 0; j < nb; ++j) z += sh.kw[j][tid];
                sh.n[tid] = z;
            }
        }
    }
    __syncthreads();
    float* st_out = st;
    if (x.pass == 1) {
        st_out = x.seg_state + ((int64_t)s * x.n_seg + seg) * plane + (int64_t)h * dim * V1;
        if (x.seg_decay != nullptr && tid == 0 && c0 == 0) x.seg_decay[((int64_t)s * x.n_seg + seg) * x.heads + h] = total;
    } else if (cut && !last_seg) {
        return;
    }
    for (int i = tid; i < dim * nv; i += 256) {
        const int d = i / nv, c = i - d * nv;
        st_out[(int64_t)d * V1 + c0 + c] = sh.s[d][c];
    }
    if (norm && tid < dim) st_out[(int64_t)tid * V1 + vdim] = sh.n[tid];
}

// Keys of 28 and 32 numbers walk: the walk's smallest form holds up to 32 of them and a piece's products grow with them (16 sequences
// of 512 tokens, 4 heads, mLSTM, walked / in pieces: 24 x 32 165 / 159 us, 32 x 32 138 / 164; retention of 64 tokens, 32 x 32: 18 / 21).
bool chunk_memory_fits(int dim, int vdim) { return dim % 4 == 0 && dim <= kChD && (dim <= 24 || dim > 32) && vdim % 4 == 0; }
int chunk_base_blocks(int n_seqs, int heads, int vdim) { return n_seqs * heads * ((vdim + kChV - 1) / kChV); }

int chunk_segments(int base_blocks, int max_seq_len, size_t fit, int* seg_len) {
    *seg_len = max_seq_len;
    // two passes cost 1.4 of one: worth it from two and a half times the blocks
    int want = std::min(296 / std::max(base_blocks, 1), max_seq_len / (2 * kChunkTokens));
    want = (int)std::min<size_t>(want, fit);
    if (want < 3) return 1;
    *seg_len = ((max_seq_len + want - 1) / want + kChunkTokens - 1) / kChunkTokens * kChunkTokens;
    return (max_seq_len + *seg_len - 1) / *seg_len;
}

int launch_chunk_memory(const ChunkMemory& m, const Batch& b, cudaStream_t st) {
    const dim3 grid(b.n_seqs * m.n_seg, m.heads, (m.vdim + kChV - 1) / kChV);
    auto run = [&](auto kernel) -> int {
        const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(ChunkShared));
        if (e != cudaSuccess) return (int)e;
        // (two blocks to an SM, often fewer of them than SMs: brought in while the angles or gates in front are worked out, two heavy ones fell on
        // one SM.  us, early / not: a sequence of 171 tokens, 16 heads 64 x 128 80 / 63; 113 and 105 tokens, 4 heads 60 x 132 59 / 46)
        return chain_launch_if(false, kernel, grid, 256, sizeof(ChunkShared), st, m, b);
    };
    return m.gates != nullptr ? run(chunk_memory_kernel<true>) : run(chunk_memory_kernel<false>);
}

}  // namespace umbs
