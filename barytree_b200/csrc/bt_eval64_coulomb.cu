// bt_eval64_coulomb.cu -- FP64 evaluation kernels: Coulomb.
#include "bt_eval64.cuh"

namespace bt {

BT_EVAL64_INSTANTIATE(K_COULOMB, false)
BT_EVAL64_INSTANTIATE_DIRECT(K_COULOMB)

}  // namespace bt
