// score16_variants.h -- the compiled forms of the 16-bit score sweep.  Each
// group is instantiated in a translation unit of its own (score16_*.cu), so
// that they compile side by side.
#pragma once
#include "pw_score16.cuh"

namespace pw {

// A kernel of the 16-bit sweep and its dynamic shared memory.
struct Score16Kernel {
    void (*kern)(Score16Args) = nullptr;
    int smem = 0;
};

// rows: the one-strip height of score16_kernel, 0 its multi-strip form (32-row
// strips, one warp an item), -1 score16_chain_kernel.
Score16Kernel score16_linear(int form, int rows, int alpha1);   // kPair128, kPair64, kPair32
Score16Kernel score16_affine(int form, int rows, int alpha1);
Score16Kernel score16_dual(bool affine, int rows, int alpha1);  // kDual

template <bool AFFINE, int FORM>
Score16Kernel score16_pick(int rows, int alpha1) {
    Score16Kernel k;
    auto one = [&](auto kern, int smem) {
        k.kern = kern;
        k.smem = smem;
    };
    switch (rows) {
        case -1: one(score16_chain_kernel<32, AFFINE, FORM>, score16_smem<32, AFFINE, FORM, true>(alpha1)); break;
        case 0: one(score16_kernel<32, AFFINE, true, FORM>, score16_smem<32, AFFINE, FORM, true>(alpha1)); break;
        case 16: one(score16_kernel<16, AFFINE, false, FORM>, score16_smem<16, AFFINE, FORM, false>(alpha1)); break;
        case 24: one(score16_kernel<24, AFFINE, false, FORM>, score16_smem<24, AFFINE, FORM, false>(alpha1)); break;
        case 32: one(score16_kernel<32, AFFINE, false, FORM>, score16_smem<32, AFFINE, FORM, false>(alpha1)); break;
        default:
            if constexpr (!AFFINE) {
                if (rows == 40)
                    one(score16_kernel<40, false, false, FORM>, score16_smem<40, false, FORM, false>(alpha1));
                else if (rows == 48)
                    one(score16_kernel<48, false, false, FORM>, score16_smem<48, false, FORM, false>(alpha1));
                else if (rows == 64)
                    one(score16_kernel<64, false, false, FORM>, score16_smem<64, false, FORM, false>(alpha1));
            }
    }
    return k;
}

}  // namespace pw
