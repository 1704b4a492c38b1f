// Matrix memories with one decay per head and token, many tokens at a time (seq_chunk.cu): S <- a S + b k v^T, o = S^T q.
#pragma once
#include "seq_internal.h"

namespace umbs {

struct ChunkMemory {
    const float* x; int64_t ld;                  // the projection: q, k, v of head h at offsets + h dim, + h dim, + h vdim of a token's row
    int qoff, koff, voff, heads, dim, vdim;
    float qscale, kscale;
    int rot_dims; const float* rot_tab;          // queries and keys turn by the table's cos | sin rows (rot_dims 0: they do not)
    const float* decay;                          // [heads]: one decay for every token, b = 1 ...
    const float* gates;                          // ... or [tokens, heads, 3]: decay a, weight b of every token (decay NULL)
    int normaliser;                              // a further value column of ones (the last one of state and output)
    float* state; int64_t state_stride;          // per (slot, head)
    float* out;                                  // fp32 [tokens, heads, vdim (+ 1)]
    // a sequence cut into segments, see retention_kernel: pass 0 none, 1 end states from zero, 2 outputs from the chained starts
    int seg_len, n_seg, pass;
    float* seg_state; float* seg_decay;          // seg_decay: products of a segment's decays (pass 1 with gates), or NULL
};

constexpr int kChunkTokens = 32;
bool chunk_memory_fits(int dim, int vdim);
// Segments of a step of this many blocks without any and this longest sequence: enough for two blocks on every SM, at most `fit`.
int chunk_segments(int base_blocks, int max_seq_len, size_t fit, int* seg_len);
int chunk_base_blocks(int n_seqs, int heads, int vdim);
int launch_chunk_memory(const ChunkMemory& m, const Batch& b, cudaStream_t st);

// seq_chunk_tc.cu, one decay per head: the 128-token pieces of the longest sequence if the tensor-core kernels take these sizes and
// addresses and `fit` states per sequence are room enough, else 0.  launch_chunk_tc (m.n_seg: that number): norm_dtype UMBS_*: every
// head's unit norm and silu gate too, results in `out`; -1: plain results in m.out.
int chunk_tc_count(const ChunkMemory& m, const Batch& b, const void* out, size_t fit);
int launch_chunk_tc(const ChunkMemory& m, const Batch& b, int norm_dtype, float eps, void* out, cudaStream_t st);

}  // namespace umbs
