// score16_affine.cu -- 16-bit score sweep: affine gap.
#define PW_SCORE_SWEEP_ONLY
#include "score16_variants.h"

namespace pw {

Score16Kernel score16_affine(int form, int rows, int alpha1) {
    switch (form) {
        case kPair64: return score16_pick<true, kPair64>(rows, alpha1);
        case kPair32: return score16_pick<true, kPair32>(rows, alpha1);
        default: return score16_pick<true, kPair128>(rows, alpha1);
    }
}

}  // namespace pw
