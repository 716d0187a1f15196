// march_reg.cuh - launch interface of the column-parallel march with its
// factors in registers (march_reg.cu), complex128.
#pragma once

#include "march_col.cuh"

namespace crk {

// Rows of a lane (the kernel's template values) for a column of nz rows on a
// cluster of `cluster` CTAs; 0 when a slice is too long for the kernel.
int reg_rows(int nz, int cluster);

// One cluster of `cluster` CTAs of 32 x terms threads per ray; every ray of
// the launch has at most `terms` Pade terms in every set, at most nz_max rows
// and the same reg_rows(nz, cluster) = rows.
cudaError_t launch_march_reg(const ColArgs& a, int n_rays, int cluster, int terms, int rows, int nz_max,
                             cudaStream_t st);

// Clusters of the launch's shape that can be resident at once (0: the
// configuration cannot run).
int reg_max_active_clusters(int cluster, int terms, int rows, int nz_max, int grids);

}  // namespace crk
