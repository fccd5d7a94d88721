// The sweeps' use of collide_mrt1: its collision operator and register budgets.
#pragma once
#include "lbm_collide_mrt1.cuh"
#include "lbm_mrt1.h"

namespace lbm {

template <> struct Collision<MK_MRT1> {
    template <int Q, class R, class P>
    __device__ __forceinline__ static R run(R (&f)[Q], const P& p) { return collide_mrt1<Q, R>(f, p); }
};

// Resident 256-thread blocks per SM (see the primary templates).  The populations are dead once their sums are
// taken, so that little or nothing spills: 12 bytes in the FP32 pull sweep, 20 in the 16-bit pair AA odd ones, 24
// to 104 in the batched sweeps, none in the others.
template <int PAT> struct SweepMinBlocks<float, 19, MK_MRT1, PAT> { static constexpr int value = PAT == PAT_PULL ? 5 : 4; };
template <int PAT> struct SweepMinBlocks<__half, 19, MK_MRT1, PAT> { static constexpr int value = 4; };
template <int PAT> struct SweepMinBlocks<__nv_bfloat16, 19, MK_MRT1, PAT> { static constexpr int value = 4; };
template <int PAT> struct SweepMinBlocks<e3m12, 19, MK_MRT1, PAT> { static constexpr int value = 4; };
template <int PAT> struct SweepMinBlocks<double, 19, MK_MRT1, PAT> { static constexpr int value = 2; };
template <int PAT> struct SweepMinBlocks<float, 27, MK_MRT1, PAT> { static constexpr int value = 3; };
template <int PAT> struct SweepMinBlocks<double, 27, MK_MRT1, PAT> { static constexpr int value = 2; };
template <> struct BatchMinBlocks<float, 19, MK_MRT1> { static constexpr int value = 4; };
template <int Q> struct BatchMinBlocks<double, Q, MK_MRT1> { static constexpr int value = 3; };

}  // namespace lbm
