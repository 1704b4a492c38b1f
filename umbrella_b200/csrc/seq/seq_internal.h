// Internal helpers shared by the translation units of libumbrella_b200_seq.so.
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <utility>

#include "../../../include/umbrella_b200.h"      // UMB_ERR_*
#include "../../../include/umbrella_b200_seq.h"

namespace umbs {
typedef umbs_batch_t Batch;

template <typename T> __device__ __forceinline__ float to_f32(T v);
template <> __device__ __forceinline__ float to_f32<float>(float v) { return v; }
template <> __device__ __forceinline__ float to_f32<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }
template <typename T> __device__ __forceinline__ T from_f32(float v);
template <> __device__ __forceinline__ float from_f32<float>(float v) { return v; }
template <> __device__ __forceinline__ __nv_bfloat16 from_f32<__nv_bfloat16>(float v) { return __float2bfloat16_rn(v); }

// Two fp32 numbers in one register pair: one instruction multiplies and adds both, each rounded as its scalar form rounds.
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pack2(float a, float b) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float2 unpack2(f32x2 v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}

void count_launches(unsigned n);

// Kernels that follow one another: one may be brought onto the SMs while the one in front of it still runs, and waits there (chain_wait,
// ahead of everything it reads or writes but a model's weights) until that one is done and its results are visible.  Every block
// waits, so a kernel is done only after all those in front of it are.  A decode step is some 80 kernels of 2 to 6 us each; launched
// one behind the other, 1.2 us of each are its launch.
// A ChainScope says that the launches are one umbs_forward's, whose products' weights were there before its first kernel.
class ChainScope {                                          // this thread's launches until the scope ends
public:
    ChainScope();
    ~ChainScope();
    ChainScope(const ChainScope&) = delete;
    ChainScope& operator=(const ChainScope&) = delete;
};
bool in_chain();
template <typename... P, typename... A>
int chain_launch_if(bool early_too, void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A&&... args) {
    cudaLaunchAttribute early{};
    early.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    early.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t c{};
    c.gridDim = grid;
    c.blockDim = block;
    c.dynamicSmemBytes = smem;
    c.stream = st;
    c.attrs = &early;
    c.numAttrs = early_too ? 1 : 0;
    return (int)cudaLaunchKernelEx(&c, kernel, std::forward<A>(args)...);
}
template <typename... P, typename... A>
int chain_launch(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A&&... args) {
    return chain_launch_if(true, kernel, grid, block, smem, st, std::forward<A>(args)...);
}
// The two halves of it, apart in a kernel that takes tensor memory behind the wait: it lets the next one in when it has it (any thread's
// chain_next counts for its block).  The products take theirs ahead of their wait: one brought onto an SM beside a block that has none yet
// could hold all of it, and each would wait for the other for good.
__device__ __forceinline__ void chain_wait_only() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void chain_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void chain_wait() {
    chain_wait_only();
    chain_next();
}

// seq_gemm_tc.cu: a word of host memory that the kernels can write, set by a block that gave up.  Every call that launches such
// a kernel looks at it first (no synchronisation) and refuses once it is set: results since then are not to be used.
int give_up_word(unsigned int** word);                      // made on the first call; an error of the runtime, or 0
int give_up_status();                                       // 0, or UMB_ERR_TIMEOUT
}  // namespace umbs
