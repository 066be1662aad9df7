// Compiled instances of the 3D iteration kernel for the labelled models
// (divergence epilogue); EXACT projection, built with the
// reference's float arithmetic (no FMA contraction, no flush to zero).
#include "variants.cuh"

namespace asets {

static const StencilVariant kVariants[] = {
    make_variant3<16, 2, 4, EPI_DIV, true>(),
    make_variant3<14, 2, 3, EPI_DIV, true>(),
    make_variant3<13, 2, 4, EPI_DIV, true>(),
    make_variant3<12, 2, 4, EPI_DIV, true>(),
    // 32-row tiles for volumes of up to 32 rows (step_cost3)
    make_variant3<16, 1, 4, EPI_DIV, true>(),
    make_variant3<12, 1, 4, EPI_DIV, true>(),
    make_variant3<10, 1, 4, EPI_DIV, true>(),
};

const StencilVariant *flow3d_exact_variants(int *count)
{
    *count = (int)(sizeof(kVariants) / sizeof(kVariants[0]));
    return kVariants;
}

}  // namespace asets
