// Host build of the two MRT collisions (lbm_collide.cuh, lbm_collide_mrt1.cuh).  Test infrastructure only.
#define __device__
#define __host__
#define __forceinline__ inline
#include <cmath>
using std::sqrt;
#include "../../lbmpy_b200/csrc/lbm_collide.cuh"
#include "../../lbmpy_b200/csrc/lbm_collide_mrt1.cuh"

using namespace lbm;

template <int Q, class R> static double run(int special, double* f, const Physics* p) {
    R g[Q];
    for (int i = 0; i < Q; ++i) g[i] = (R)f[i];
    const R om = special ? collide_mrt1<Q, R>(g, *p) : collide_mrt<Q, R>(g, *p);
    for (int i = 0; i < Q; ++i) f[i] = g[i];
    return om;
}

extern "C" double host_mrt(int q, int special, int fp32, double* f, const Physics* p) {
    if (q == 19) return fp32 ? run<19, float>(special, f, p) : run<19, double>(special, f, p);
    return fp32 ? run<27, float>(special, f, p) : run<27, double>(special, f, p);
}
