// gmi_wall_kernel.hpp -- host interface of the FP64 wall pair sum.
#pragma once

#include "gmi_context.hpp"

namespace gmi {

// out = M_ss F above the wall z = 0 (radius and viscosity 1) for targets
// [tgt_start, tgt_start + n_tgt) of the n_src segments.
struct WallSum {
    const double *x, *f;  // AoS positions and loads (6 values)
    int tgt_start, n_tgt, n_src;
    double *out;
    double *partial;  // wall_splits() * 6 n_tgt values when there are several splits, or when out overlaps an
                      // input (a last kernel then writes out); else null
};

int wall_splits(int n_tgt, int n_src, int sm_count);
// One or two launches (*launched counts them).
gmi_status launch_wall_fp64(cudaStream_t stream, int sm_count, const WallSum &a, int *launched);

}  // namespace gmi
