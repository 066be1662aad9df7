// x/c for a divisor that stays the same through a launch, rounded to nearest
// as the division rounds it.
#pragma once

#include <cmath>

namespace asets {

// From 1/c = r + r_lo (r rounded to nearest): q = x*r + x*r_lo is within an
// ulp of the quotient (half an ulp of its own rounding, 2^-50 of one for the
// terms), so Markstein's correction (Markstein, "Computation of elementary
// functions on the IBM RISC System/6000", 1990) with the exact residual x -
// q*c rounds it correctly.  Zero keeps its sign; exponents where a term could
// leave the normal range (and non-finite x) take the division.  Double
// precision only, whose operations are slow here: four against some twelve.  In
// single precision that would gain nothing on the division.
__device__ __forceinline__ double div_markstein(double x, double c, double r, double r_lo, unsigned int span)
{
    const int e = __double2hiint(x) & 0x7ff00000;
    if ((unsigned int)(e - 0x10000000) < span) {
        double q = __fma_rn(x, r, __dmul_rn(x, r_lo));
        const double d = __fma_rn(-q, c, x);
        return __fma_rn(d, r, q);
    }
    return x == 0.0 ? __dmul_rn(x, r) : __ddiv_rn(x, c);
}

template <class T>
struct DivConst {
    T r, r_lo;
    unsigned int span;  // exponents the correction holds for (0: none)
    int exact;          // c a power of two: x*r is x/c, rounded alike

    void set(T c)
    {
        r = (T)1 / c;
        // the residual 1 - r*c is exact
        r_lo = (T)(std::fma(-(double)r, (double)c, 1.0) / (double)c);
        int exp = 0;
        const double frac = std::fabs(std::frexp((double)c, &exp));
        exact = frac == 0.5 && std::isnormal(r) && std::isnormal(c);
        // 2^-767 <= |x| < 2^769 for an ordinary c; the correction's proof
        // leaves out a divisor whose significand is all ones
        span = (std::isnormal((double)c) && std::abs(exp) < 200 && frac < 1.0 - 0x1p-53) ? 0x60000000u : 0u;
    }
    __device__ __forceinline__ T operator()(T x, T c) const
    {
        if constexpr (sizeof(T) == 8)
            return exact ? __dmul_rn(x, r) : div_markstein(x, c, r, r_lo, span);
        else
            return exact ? __fmul_rn(x, r) : __fdiv_rn(x, c);
    }
};

}  // namespace asets
