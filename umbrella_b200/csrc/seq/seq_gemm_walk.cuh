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

}  // namespace umbs
