// score16_linear.cu -- 16-bit score sweep: linear gap.
#define PW_SCORE_SWEEP_ONLY
#include "score16_variants.h"

namespace pw {

Score16Kernel score16_linear(int form, int rows, int alpha1) {
    switch (form) {
        case kPair64: return score16_pick<false, kPair64>(rows, alpha1);
        case kPair32: return score16_pick<false, kPair32>(rows, alpha1);
        default: return score16_pick<false, kPair128>(rows, alpha1);
    }
}

}  // namespace pw
