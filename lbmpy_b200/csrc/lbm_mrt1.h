// Launchers of the MRT sweeps whose moments of order >= 3 relax with rate 1 (lbm_mrt1.cuh).  The staged
// sweep, the boundary pre-pass and the setters are those of the general MRT family.
#pragma once
#include "lbm_dispatch.h"

namespace lbm {

SweepLauncher sweep_q19_mrt1(int store, int pat);
SweepLauncher sweep_pair_q19_mrt1(int store, int pat);
SweepLauncher sweep_quad_q19_mrt1(int store, int pat);
BatchLauncher batched_q19_mrt1(int store, int pat);
SparseLauncher sparse_q19_mrt1(int store);

SweepLauncher sweep_q27_mrt1(int store, int pat);
SweepLauncher sweep_pair_q27_mrt1(int store, int pat);
BatchLauncher batched_q27_mrt1(int store, int pat);
SparseLauncher sparse_q27_mrt1(int store);

}  // namespace lbm
