// Host build of launch_chained (lbmpy_b200/csrc/lbm_launch.h) over a stand-in for the runtime's launch call,
// which fails on demand and, like the runtime, also leaves its error in the last-error slot.
#include "../../lbmpy_b200/csrc/lbm_launch.h"

static cudaError_t answer, slot;
static unsigned grid_x;
static int attributes;

extern "C" cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void*, void**) {
    grid_x = c->gridDim.x;
    attributes = c->numAttrs;
    if (answer != cudaSuccess) slot = answer;
    return answer;
}
extern "C" cudaError_t cudaGetLastError() {
    const cudaError_t e = slot;
    slot = cudaSuccess;
    return e;
}

static void kernel(int, double) {}

// The launch's result; *left: what it left in the last-error slot.
extern "C" int host_launch(int fail, int* left, int* seen) {
    answer = (cudaError_t)fail;
    slot = cudaSuccess;
    const int e = lbm::launch_chained(&kernel, dim3(7), dim3(32), 0, nullptr, 3, 1.5f);
    *left = slot;
    *seen = int(grid_x) * 10 + attributes;
    return e;
}
