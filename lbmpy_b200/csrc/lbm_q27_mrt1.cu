// Kernel instantiations: D3Q27, MRT with every moment of order >= 3 relaxed by 1 (FP64 / FP32 storage, pull
// and AA, as the general D3Q27 MRT family).
#include "lbm_mrt1.cuh"

namespace lbm {

namespace {
template <class S, class R> SweepLauncher pick_cell(int pat) {
    switch (pat) {
        case PAT_PULL: return &launch_sweep<S, R, 27, MK_MRT1, PAT_PULL>;
        case PAT_AA_EVEN: return &launch_sweep<S, R, 27, MK_MRT1, PAT_AA_EVEN>;
        case PAT_AA_ODD: return &launch_sweep<S, R, 27, MK_MRT1, PAT_AA_ODD>;
    }
    return nullptr;
}
}  // namespace

SweepLauncher sweep_q27_mrt1(int store, int pat) {
    if (store == ST_F64) return pick_cell<double, double>(pat);
    if (store == ST_F32) return pick_cell<float, float>(pat);
    return nullptr;
}

SweepLauncher sweep_pair_q27_mrt1(int store, int pat) {
    if (store == ST_F32) return pick_pair_pattern<float, 27, MK_MRT1>(pat);
    return nullptr;
}

BatchLauncher batched_q27_mrt1(int store, int pat) {
    if (store == ST_F32) return pick_batched_pattern<float, float, 27, MK_MRT1>(pat);
    return nullptr;
}

SparseLauncher sparse_q27_mrt1(int store) {
    if (store == ST_F64) return &launch_sparse<double, double, 27, MK_MRT1>;
    if (store == ST_F32) return &launch_sparse<float, float, 27, MK_MRT1>;
    return nullptr;
}

}  // namespace lbm
