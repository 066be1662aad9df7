// Compiled instances of the 3D iteration kernel for the binary model; EXACT
// projection, built with the reference's float arithmetic (no FMA
// contraction, no flush to zero).
#include "variants.cuh"

namespace asets {

static const StencilVariant kVariants[] = {
    make_variant3<16, 2, 3, EPI_BINARY, true>(),
    make_variant3<13, 2, 3, EPI_BINARY, true>(),
    make_variant3<12, 2, 3, EPI_BINARY, true>(),
};

const StencilVariant *binary3d_exact_variants(int *count)
{
    *count = (int)(sizeof(kVariants) / sizeof(kVariants[0]));
    return kVariants;
}

}  // namespace asets
