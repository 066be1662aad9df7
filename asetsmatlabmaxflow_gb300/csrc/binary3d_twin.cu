// Compiled instances of the 3D iteration kernel for the binary Matlab twin in
// single precision (mtwin.cu), built with IEEE arithmetic.
#include "variants.cuh"

namespace asets {

static const StencilVariant kVariants[] = {
    make_variant3<16, 2, 3, EPI_TWIN, true>(),
    make_variant3<14, 2, 3, EPI_TWIN, true>(),
    make_variant3<13, 2, 3, EPI_TWIN, true>(),
    make_variant3<12, 2, 3, EPI_TWIN, true>(),
};

const StencilVariant *binary3d_twin_variants(int *count)
{
    *count = (int)(sizeof(kVariants) / sizeof(kVariants[0]));
    return kVariants;
}

}  // namespace asets
