// pdl.cuh — programmatic dependent launch: a kernel of the step's chain may start while
// the one before it drains, and waits itself for that one's results.
//
// Every kernel launched with pdl_launch calls pdl_wait() before it touches anything
// an earlier kernel of the stream writes (or reads what it will overwrite); what comes
// before may only read constants (twiddles, tensor tables).  The wait returns when the
// earlier kernel has completed, which by its own wait covers all before it.
//
// No kernel releases its dependents before it ends: with griddepcontrol.launch_dependents
// at the top (before or after the wait) the next kernels' blocks sit in the running
// kernel's SMs.  Us per pass with plain launches, with that, and as it is: 512 x 512
// FP32 Heun x 40 2454 / 2920 / 2360, 300 x 180 x 5 FP32 DP45 x 6 2923 / 2676 / 2477,
// 1024 x 512 x 16 FP32 DP45 x 4 28930 / 31204 / 28688; 250 x 100 FP64 RK4 x 20 - / 2209 /
// 1364.
#pragma once

#include <cuda_runtime.h>

#include <utility>

namespace fm {

__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Bring [p, p + bytes) into L1: one plain load per 128-byte line, spread over the
// block's threads, whose results nobody waits for.
__device__ __forceinline__ void warm_lines(const void *p, int bytes) {
    for (int o = threadIdx.x * 128; o < bytes; o += blockDim.x * 128) {
        unsigned v;
        asm volatile("ld.global.u32 %0, [%1];" : "=r"(v) : "l"((const char *)p + o));
        static_cast<void>(v);
    }
}

template <typename... P, typename... A>
inline cudaError_t pdl_launch(void (*kern)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A &&...args) {
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kern, std::forward<A>(args)...);
}

}  // namespace fm
