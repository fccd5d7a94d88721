// Host build of the wall words (lbmpy_b200/csrc/lbm_walls.cuh).  Test infrastructure only.
#define __device__
#define __host__
#define __forceinline__ inline
#define __noinline__
#include <cmath>
#include "../../lbmpy_b200/csrc/lbm_walls.cuh"

using namespace lbm;

template <int Q> static void run(const Grid& g, uint32_t* words) {
    for (int z = 0; z < g.nz; ++z)
        for (int y = 0; y < g.ny; ++y)
            for (int x = 0; x < g.nx; ++x) words[x + g.nx * (y + g.ny * z)] = wall_word_of_flags<Q>(g, x, y, z);
}

// Wall word of every interior cell; periodic: bit 0 x, bit 1 y, bit 2 z.
extern "C" void host_wall_words(int q, int nx, int ny, int nz, int periodic, const uint8_t* flags, uint32_t* words) {
    Grid g = {};
    g.nx = nx; g.ny = ny; g.nz = nz;
    g.periodic = periodic;
    g.flags = flags;
    g.fsy = nx + 2;
    g.fsz = (nx + 2) * (ny + 2);
    if (q == 19) run<19>(g, words); else run<27>(g, words);
}
