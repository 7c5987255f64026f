// bt_eval64.h -- launchers of the FP64 evaluation kernels of one kernel type
// (bt_eval64.cuh, instantiated in bt_eval64_*.cu; the kernel types with short
// forms have a translation unit each, because their compilation dominates
// the build).
#pragma once

#include "bt_device.h"

namespace bt {

// FAR: Yukawa calls whose exponentials can leave the short form's range.
template <int KT, bool FAR = false>
void eval_targets_kt(bool hermite, const EvalTargetsArgs &a, cudaStream_t st);
template <int KT, bool FAR = false>
void eval_grids_kt(const EvalGridsArgs &a, cudaStream_t st);
template <int KT>
void direct_kt(int nt, int ns, int parts, const double *tx, const double *ty, const double *tz, const double *sx,
               const double *sy, const double *sz, const double *sq, double kp, double kp2, double *out,
               cudaStream_t st);

}  // namespace bt
