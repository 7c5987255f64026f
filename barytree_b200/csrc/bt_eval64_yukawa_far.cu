// bt_eval64_yukawa_far.cu -- FP64 evaluation kernels: Yukawa with exponentials
// beyond the short form's range.
#include "bt_eval64.cuh"

namespace bt {

BT_EVAL64_INSTANTIATE(K_YUKAWA, true)

}  // namespace bt
