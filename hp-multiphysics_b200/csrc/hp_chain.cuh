// Kernels of one update, each started under the end of the one before it (programmatic dependent
// launch). A kernel of such a chain lets the next one's CTAs start as soon as all of its own have
// (chain_next), reads only what no kernel of an update writes -- tables, connectivity, geometry --
// until the kernel before it is complete (chain_wait), and writes nothing before that. Launched
// without the attribute both do nothing. What it saves is launch latency and the first loads, 0.5 to 1
// us a kernel (figures at the launches). A chain begins with an ordinary launch, and whatever does not
// know the kernel before it launches an ordinary one. Only the vertex kernels of small p = 1 levels and
// the assembly after the line kernel are chained: the preconditioner's phases and the persistent line
// kernel after them lose what they gain (p = 6 cavity, 2 sweeps with all of it chained 6640 us against
// 6287; an FP32-smoothed solve 830 ms against 782), since their CTAs then sit on the SMs early.
#pragma once
#include <cuda_runtime.h>

namespace hpb {

__device__ __forceinline__ void chain_next() { asm volatile("griddepcontrol.launch_dependents;"); }
__device__ __forceinline__ void chain_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// chained: the kernel before this one on the stream is one of the chain
template <typename... K, typename... A>
void launch_chained(int chained, void (*kernel)(K...), unsigned grid, unsigned block, size_t smem, cudaStream_t st,
                    A... args) {
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = &at;
    cfg.numAttrs = chained ? 1 : 0;
    (void)cudaLaunchKernelEx(&cfg, kernel, static_cast<K>(args)...);  // an error is cudaGetLastError's
}

}  // namespace hpb
