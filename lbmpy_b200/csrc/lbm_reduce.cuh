// FP64 conserved sums (lbm_reduce_conserved) for every stencil, storage type and pattern.
#pragma once
#include "lbm_kernels.cuh"

namespace lbm {

// ------------------------------------------------------------------ FP64 conserved sums
// Per-block partial sums of mass, momentum (rho_ref * u, force-shifted) and kinetic energy over
// fluid cells; k_reduce_finish adds the partials in a fixed order (deterministic).
constexpr int RED_THREADS = 256;

template <class S, int Q, int PAT>
__global__ void __launch_bounds__(RED_THREADS) k_reduce_partial(const MacroArgs a, double* partial) {
    using A = Access<PAT>;
    const Grid& g = a.g;
    double acc[5] = {0, 0, 0, 0, 0};
    const long long ncell = (long long)g.nx * g.ny * g.nz;
    for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < ncell;
         c += (long long)gridDim.x * blockDim.x) {
        const int x = (int)(c % g.nx);
        const int y = (int)((c / g.nx) % g.ny);
        const int z = (int)(c / ((long long)g.nx * g.ny));
        if (g.flags != nullptr && (g.flags[(x + 1) + (y + 1) * g.fsy + (z + 1) * g.fsz] & FLAG_TYPE_MASK)) continue;
        NbrOffsets nb;
        nb.init(g, x, y, z);
        const int cell = (x + 1) + (y + 1) * g.sy + (z + 1) * g.sz;
        const S* src = static_cast<const S*>(a.pdfs);
        double f[Q];
#pragma unroll
        for (int i = 0; i < Q; ++i) {
            const int off = nb.off(A::template woff<Q>(i, 0), A::template woff<Q>(i, 1), A::template woff<Q>(i, 2));
            f[i] = Conv<S, double>::ld(at(src, A::template wslot<Q>(i) * g.sq, cell + off));
        }
        Macro<Q, double> m = conserved<Q, double>(f, a.p, false);
        if (a.p.force_model != FM_NONE) {
            const double h = 0.5 / m.rho_ref;
            m.ux += h * a.p.force[0]; m.uy += h * a.p.force[1]; m.uz += h * a.p.force[2];
        }
        acc[0] += m.rho;
        acc[1] += m.rho_ref * m.ux;
        acc[2] += m.rho_ref * m.uy;
        acc[3] += m.rho_ref * m.uz;
        acc[4] += 0.5 * m.rho * (m.ux * m.ux + m.uy * m.uy + m.uz * m.uz);
    }
    __shared__ double sh[5][RED_THREADS / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int k = 0; k < 5; ++k) {
        double v = acc[k];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
        if (lane == 0) sh[k][warp] = v;
    }
    __syncthreads();
    if (threadIdx.x < 5) {
        double v = 0;
        for (int w = 0; w < RED_THREADS / 32; ++w) v += sh[threadIdx.x][w];
        partial[blockIdx.x * 5 + threadIdx.x] = v;
    }
}

// One warp per sum: lane l adds the partials l, l + 32, ... and the lanes are added in a fixed tree, so the
// result does not depend on timing.  Bound by the latency of the loads, which are all in flight at once
// (one thread per sum, adding 592 partials one after another, took 21 us on B200, a tenth of a monitored
// 64^3 FP64 step).
static __global__ void __launch_bounds__(160) k_reduce_finish(const double* partial, int nblocks, double* out) {
    const int k = threadIdx.x >> 5, lane = threadIdx.x & 31;
    double v = 0;
#pragma unroll 8
    for (int b = lane; b < nblocks; b += 32) v += partial[b * 5 + k];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if (lane == 0) out[k] = v;
}

}  // namespace lbm
