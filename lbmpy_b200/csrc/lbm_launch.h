// Launch of the kernels that begin with chain_wait() (lbm_common.cuh).
#pragma once
#include <cuda_runtime.h>

namespace lbm {

// The kernel may start while the kernel before it in the stream still runs, and waits for it there.  A failed
// launch leaves no error behind: the runtime's last-error slot is shared with the library's other launches
// and with the caller's own checks, which would report it as theirs.
template <class... KA, class... A>
cudaError_t launch_chained(void (*kernel)(KA...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, const A&... args) {
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t c = {};
    c.gridDim = grid;
    c.blockDim = block;
    c.dynamicSmemBytes = smem;
    c.stream = s;
    c.attrs = &attr;
    c.numAttrs = 1;
    const cudaError_t e = cudaLaunchKernelEx(&c, kernel, KA(args)...);
    if (e != cudaSuccess) cudaGetLastError();
    return e;
}

}  // namespace lbm
