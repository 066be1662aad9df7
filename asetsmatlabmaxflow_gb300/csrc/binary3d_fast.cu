// Compiled instances of the 3D iteration kernel for the binary model; fast
// projection, built with FMA contraction and flush to zero (held to the
// parity tolerance, not bit-exactness).
#include "variants.cuh"

namespace asets {

// One kernel per tile width, for the cold start (pt and u in one array) and
// for a given start; the widths whose items and waves fit a volume best differ
// (pick_split3; for a batch's group batch_width3), the ring depth is the one
// that measured fastest.
static const StencilVariant kCold[] = {
    make_variant3<14, 2, 3, EPI_COLD, false>(),
    make_variant3<16, 2, 3, EPI_COLD, false>(),
    make_variant3<13, 2, 3, EPI_COLD, false>(),
    make_variant3<12, 2, 3, EPI_COLD, false>(),
};

static StencilVariant with_cold(StencilVariant v, const StencilVariant *c)
{
    v.cold = c;
    return v;
}

static const StencilVariant kVariants[] = {
    with_cold(make_variant3<14, 2, 3, EPI_BINARY, false>(), &kCold[0]),
    with_cold(make_variant3<16, 2, 3, EPI_BINARY, false>(), &kCold[1]),
    with_cold(make_variant3<13, 2, 3, EPI_BINARY, false>(), &kCold[2]),
    with_cold(make_variant3<12, 2, 3, EPI_BINARY, false>(), &kCold[3]),
};

const StencilVariant *binary3d_fast_variants(int *count)
{
    *count = (int)(sizeof(kVariants) / sizeof(kVariants[0]));
    return kVariants;
}

}  // namespace asets
