// Kernel instantiations: D3Q19, MRT with every moment of order >= 3 relaxed by 1; every storage type and
// pattern of the one-cell sweep, the pair and quad sweeps, the batched and the sparse sweep.
#include "lbm_mrt1.cuh"

namespace lbm {

SweepLauncher sweep_q19_mrt1(int store, int pat) {
    switch (store) {
        case ST_F64: return pick_sweep_pattern<double, double, 19, MK_MRT1>(pat);
        case ST_F32: return pick_sweep_pattern<float, float, 19, MK_MRT1>(pat);
        case ST_F16: return pick_sweep_pattern<__half, float, 19, MK_MRT1>(pat);
        case ST_BF16: return pick_sweep_pattern<__nv_bfloat16, float, 19, MK_MRT1>(pat);
        case ST_E3M12: return pick_sweep_pattern<e3m12, float, 19, MK_MRT1>(pat);
    }
    return nullptr;
}

SweepLauncher sweep_pair_q19_mrt1(int store, int pat) {
    switch (store) {
        case ST_F32: return pick_pair_pattern<float, 19, MK_MRT1>(pat);
        case ST_F16: return pick_pair_pattern<__half, 19, MK_MRT1>(pat);
        case ST_BF16: return pick_pair_pattern<__nv_bfloat16, 19, MK_MRT1>(pat);
        case ST_E3M12: return pick_pair_pattern<e3m12, 19, MK_MRT1>(pat);
    }
    return nullptr;
}

SweepLauncher sweep_quad_q19_mrt1(int store, int pat) {
    switch (store) {
        case ST_F16: return pick_quad_pattern<__half, 19, MK_MRT1>(pat);
        case ST_BF16: return pick_quad_pattern<__nv_bfloat16, 19, MK_MRT1>(pat);
        case ST_E3M12: return pick_quad_pattern<e3m12, 19, MK_MRT1>(pat);
    }
    return nullptr;
}

BatchLauncher batched_q19_mrt1(int store, int pat) {
    if (store == ST_F64) return pick_batched_pattern<double, double, 19, MK_MRT1>(pat);
    if (store == ST_F32) return pick_batched_pattern<float, float, 19, MK_MRT1>(pat);
    return nullptr;
}

SparseLauncher sparse_q19_mrt1(int store) {
    if (store == ST_F64) return &launch_sparse<double, double, 19, MK_MRT1>;
    if (store == ST_F32) return &launch_sparse<float, float, 19, MK_MRT1>;
    return nullptr;
}

}  // namespace lbm
