// Library-internal host helpers shared by the translation units of libumbrella_b200.so.
#pragma once
#include <cuda_runtime.h>

#include "../../include/umbrella_b200.h"

#include <utility>

namespace umb {
// Programmatic dependent launch (PDL): every kernel of the forward chain is launched with the
// programmatic-stream-serialization attribute, so its CTAs may start (barrier init, TMEM allocation,
// weight TMA + dequantisation -- nothing that depends on the predecessor) while the stream predecessor
// is still draining.  Each such kernel executes griddepcontrol.wait before touching global memory a
// predecessor wrote, and before completing (transitivity of the chain).  UMB_PDL=0 disables it.
bool pdl_enabled();
// UMB_SYNC_DEBUG=1: synchronise after every launch and name the kernel that faulted (debugging aid)
bool sync_debug();
cudaError_t sync_debug_check(const char* name, dim3 grid, dim3 block, cudaStream_t st, cudaError_t launch_rc);
template <typename... KArgs, typename... Args>
inline cudaError_t launch_pdl(const char* name, void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem,
                              cudaStream_t st, Args&&... args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl_enabled() ? 1 : 0;
    const cudaError_t rc = cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
    return sync_debug() ? sync_debug_check(name, grid, block, st, rc) : rc;
}
#define UMB_LAUNCH_PDL(kernel, ...) do { cudaError_t e__ = umb::launch_pdl(#kernel, kernel, __VA_ARGS__); if (e__ != cudaSuccess) return (int)e__; } while (0)
// every host entry point reports the kernels it enqueued (umb_launch_count)
void count_launches(unsigned n);
// 4 bytes of host memory for the process, shared by its devices, streams and threads, that a block which gave up on a bounded wait sets: results since then are
// not to be used, workspaces may hold words that are not theirs.  Made on the first call; an error of the runtime, or 0.
int give_up_word(unsigned int** word);
int give_up_status();                                       // 0, or UMB_ERR_TIMEOUT
// gemm_wide.cu: AWQ products of 129 to 512 token rows by pairs of SMs, with a workspace of awq_wide_ws_bytes() bytes
struct GemmParams;
size_t awq_wide_ws_bytes(int M, int N_total);
int launch_awq_wide(const void* x, int64_t ldx, const GemmParams& p, cudaStream_t st);
// gemm.cu: umb_awq_gemm_f16 of up to 512 token rows
int awq_gemm_rows(const void* x, int64_t ldx, const void* packed, void* y, int64_t ldy, int M, int K, int N_total, const umb_epilogue_t* epi,
                  void* workspace, size_t workspace_bytes, cudaStream_t st);
// number of SMs of the current device (cached)
int sm_count();
// graph-replay variants (device-resident prefix length), used by the native forward driver
int embedding_dyn(const int64_t* ids_base, const int32_t* n_dev, int offset, const void* table, void* y, int rows,
                  int hidden, cudaStream_t st);
int rope_append_dyn(const void* qkv, int64_t ld_qkv, void* q_out, void* k_cache, void* v_cache, const void* cos,
                    const void* sin, const int64_t* position_base, const int32_t* n_dev, int offset, int qo, int Hq,
                    int Hkv, int D, int64_t kv_tok_stride, int64_t kv_head_stride, cudaStream_t st);
}  // namespace umb
