// Chained kernel launches.
#pragma once
#include <cuda_runtime.h>

namespace ck {

// Launch of a kernel that follows another on its stream and may be set up
// while that one still runs (programmatic dependent launch; the same edge in a
// captured graph).  Such a kernel begins with chain_begin: nothing is read or
// written before it, by any of its threads, so that everything earlier on the
// stream is complete when it returns; it then lets the next one be set up.
// The list build's ten kernels run one after the other, each short beside the gap
// before it: whole calls of one configuration with a 12/10/4 set, without and with it,
// FP64 8191 atoms 875 -> 858 us, 3000 417 -> 403, 1024 247 -> 239, 333 188 -> 183; mixed
// 470 -> 450, 281 -> 262, 200 -> 193.
template <class... P, class... A>
inline void launch_chained(void (*kernel)(P...), dim3 grid, unsigned block, size_t smem, cudaStream_t st, A... args) {
    cudaLaunchAttribute at = {};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, kernel, P(args)...);
}
__device__ __forceinline__ void chain_begin() {
    asm volatile("griddepcontrol.wait;\n griddepcontrol.launch_dependents;" ::: "memory");
}

}  // namespace ck
