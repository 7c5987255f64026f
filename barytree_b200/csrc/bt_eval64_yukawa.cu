// bt_eval64_yukawa.cu -- FP64 evaluation kernels: Yukawa.
#include "bt_eval64.cuh"

namespace bt {

BT_EVAL64_INSTANTIATE(K_YUKAWA, false)
BT_EVAL64_INSTANTIATE_DIRECT(K_YUKAWA)

}  // namespace bt
