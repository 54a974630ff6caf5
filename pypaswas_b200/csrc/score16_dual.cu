// score16_dual.cu -- 16-bit score sweep: the dual-lane form.
#define PW_SCORE_SWEEP_ONLY
#include "score16_variants.h"

namespace pw {

Score16Kernel score16_dual(bool affine, int rows, int alpha1) {
    return affine ? score16_pick<true, kDual>(rows, alpha1) : score16_pick<false, kDual>(rows, alpha1);
}

}  // namespace pw
