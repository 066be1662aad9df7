// Compiled instances of the 3D iteration kernel for the labelled models
// (divergence epilogue); fast projection, built with FMA
// contraction and flush to zero (held to the parity tolerance, not bit-exactness).
#include "variants.cuh"

namespace asets {

static const StencilVariant kVariants[] = {
    make_variant3<16, 2, 4, EPI_DIV, false>(),
    make_variant3<14, 2, 4, EPI_DIV, false>(),
    make_variant3<13, 2, 4, EPI_DIV, false>(),
    make_variant3<12, 2, 4, EPI_DIV, false>(),
    // 32-row tiles for volumes of up to 32 rows (step_cost3)
    make_variant3<16, 1, 4, EPI_DIV, false>(),
    make_variant3<12, 1, 4, EPI_DIV, false>(),
    make_variant3<10, 1, 4, EPI_DIV, false>(),
};

const StencilVariant *flow3d_fast_variants(int *count)
{
    *count = (int)(sizeof(kVariants) / sizeof(kVariants[0]));
    return kVariants;
}

}  // namespace asets
