// Order between the kernels that write weights and the decode-sized ones that read weights early.
//
// A streaming product is launched with programmatic stream serialization and fetches its weights before it waits for the kernel
// ahead of it, whose writes are sure to be visible only after that wait.  So the launch behind a kernel that wrote weights does
// without the attribute: it starts once that kernel is complete, and everything later follows it.
#pragma once

#include "common.cuh"

#include <utility>

namespace t81b200 {

// launch_behind: a kernel that starts while the one ahead ends (programmatic stream serialization).  It touches no global memory before
// its griddepcontrol.wait, behind which all of that kernel's writes are visible.  wait_for_kernel_ahead is that wait as a first
// statement, and lets the kernel's own successor start (there, or with `release` false as its blocks end).  So the order of memory is the stream's, and what overlaps is the launch
// (1 to 2 us between two short kernels).  Not for kernels of many warps behind long ones, whose SMs they wait on: the absmax
// reduction behind a weight gradient cost that 2 %.
__device__ __forceinline__ void wait_for_kernel_ahead(bool release = true) {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if (release) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
template <typename... Params, typename... Args>
cudaError_t launch_behind(void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, Args &&...args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
}

// Notes that a kernel just launched on the stream writes weights (limbs or codes).
void note_weights_written(cudaStream_t st);
// Whether that is so for a stream on which no streaming product has been launched since; takes the note away.
bool take_weights_written(cudaStream_t st);

}  // namespace t81b200
