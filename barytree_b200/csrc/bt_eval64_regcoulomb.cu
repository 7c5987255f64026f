// bt_eval64_regcoulomb.cu -- FP64 evaluation kernels: regularized Coulomb.
#include "bt_eval64.cuh"

namespace bt {

BT_EVAL64_INSTANTIATE(K_REGCOULOMB, false)
BT_EVAL64_INSTANTIATE_DIRECT(K_REGCOULOMB)

}  // namespace bt
