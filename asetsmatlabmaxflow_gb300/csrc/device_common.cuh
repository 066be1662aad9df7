// Device-side building blocks shared by the solver kernels: TMA tiled loads,
// mbarriers with bounded waits, and the reference's float arithmetic.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "kernel_args.h"

namespace asets {

// Budget of every spin-wait in these kernels: a tile load takes
// microseconds, so one second means the copy is lost.
constexpr unsigned long long kWaitBudgetNs = 1000000000ull;

__device__ __forceinline__ unsigned long long global_timer_ns()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// ---------------------------------------------------------------- mbarrier
__device__ __forceinline__ uint32_t smem_addr(const void *p)
{
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// The first 128-byte boundary in a shared array, by arithmetic on the array
// itself, so that the compiler keeps seeing shared addresses (32-bit accesses
// instead of generic ones).
__device__ __forceinline__ unsigned char *smem_align128(unsigned char *p)
{
    return p + ((128u - (smem_addr(p) & 127u)) & 127u);
}

__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count));
}

__device__ __forceinline__ void mbar_fence_init()
{
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t *bar, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)),
                 "r"(bytes)
                 : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t *bar, uint32_t phase)
{
    uint32_t ok;
    // the thread may sleep in try_wait for up to the hint (ns) before retrying
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_addr(bar)), "r"(phase), "r"(20000u)
        : "memory");
    return ok != 0;
}

// Wait for `phase` of `bar` to complete, giving up after kWaitBudgetNs.
// Returns false on timeout.  `abort_flag` (shared) short-cuts the wait once
// another thread of the block has already given up.
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t *bar, uint32_t phase,
                                                  volatile int *abort_flag)
{
    if (mbar_try_wait(bar, phase))
        return true;
    const unsigned long long t0 = global_timer_ns();
    while (true) {
        if (mbar_try_wait(bar, phase))
            return true;
        if (*abort_flag)
            return false;
        if (global_timer_ns() - t0 > kWaitBudgetNs) {
            *abort_flag = 1;
            return false;
        }
    }
}

// ---------------------------------------------------------------- TMA
// 4D tiled load of one box into shared memory, completing on `bar`.
// Coordinates: {row, col, plane, label}; out-of-range elements read as 0.
// The row coordinate must be a multiple of 4 (16 bytes of fp32).
__device__ __forceinline__ void tma_load_4d(void *smem_dst, const CUtensorMap *map, int c0, int c1,
                                            int c2, int c3, uint64_t *bar)
{
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%2, %3, %4, %5}], [%6];" ::"r"(smem_addr(smem_dst)),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(c2), "r"(c3),
        "r"(smem_addr(bar))
        : "memory");
}

// Tensor maps in global memory (a batch's) are read through a proxy of their
// own, which an earlier copy to the same place does not reach by itself: each
// block acquires a map it uses before its first load through it.  A launch that
// finds other maps at the address of the one before (another layout's) would
// else be free to load through the old ones.  Maps among a launch's parameters
// (BatchArgs::maps) need no fence.
__device__ __forceinline__ void tensormap_acquire(const CUtensorMap *map)
{
    asm volatile("fence.proxy.tensormap::generic.acquire.sys [%0], 128;" ::"l"(
        reinterpret_cast<uint64_t>(map)));
}
// The maps of parity par of an item's problem whose bits are set (HALO: Slot,
// TILE: TileSlot), one a lane of the producer's warp.  Nothing writes maps while a
// launch runs, so a block acquires those of its first item, and again only where
// the problem is another one (s_maps: the last acquired, -1 none).  Called between
// the two barriers that hand out an item, before any of its values is held:
// further down, the fence cost registers (100 iterations of Ishikawa 1024^2 L = 8
// took 7.6 ms, 6.7 here; binary 256^3 16.0, 14.8).
constexpr unsigned int kHaloMaps2D =
    1u << SL_BR | 1u << SL_BS | 1u << SL_S0 | 1u << SL_S1 | 1u << SL_S2 | 1u << SL_ALPHA;
constexpr unsigned int kTileMapsBinary = 1u << TS_S1 | 1u << TS_S2 | 1u << TS_CS | 1u << TS_CT;
template <unsigned int HALO, unsigned int TILE>
__device__ __forceinline__ void tensormaps_acquire(const BatchArgs &B, int item, int par, int *s_maps)
{
    if (B.own_maps)
        return;
    const int problem = B.item_problem[item], maps = 2 * problem + par;
    if (*s_maps == maps)
        return;
    const ProblemDesc &P = B.probs[problem];
    const unsigned int lane = threadIdx.x & 31;
    if ((HALO | TILE << NUM_SLOTS) >> lane & 1u)
        tensormap_acquire(lane < NUM_SLOTS ? &P.halo[par][lane] : &P.tile[par][lane - NUM_SLOTS]);
    __syncwarp();
    if (lane == 0)
        *s_maps = maps;
}

// The maps through which a problem of the launch is loaded.
__device__ __forceinline__ const TensorMaps &tensormaps(const BatchArgs &B, const ProblemDesc &P)
{
    return B.own_maps ? B.maps : P;
}

// ---------------------------------------------------------------- arithmetic
// The kernels are compiled with --fmad=false, so `a*b + c` is a rounded
// multiply followed by a rounded add, as in the reference's SSE code.

// |p(x)| -> gk of projStep (maxflow/asetsBinaryMF3D_mex.c:317-331) for the
// face sum s2 = sum of squared face flows.  EXACT forms the sum and the root
// in double with the reference's order; the fast path uses float.
template <bool EXACT>
struct Proj;

// The reference's norm rounded to float, fpt = (float)sqrt(0.5 * s) with s
// the double sum of the N squared face flows in order, computed in float.
// The exact sum of squares is formed as an unevaluated pair hi + lo (each
// square split exactly by FMA, the sums by TwoSum -- Knuth's error-free
// addition -- with the error terms added into lo; |hi + lo - S| <= 2^-40 S
// for N <= 6), renormalised so that |lo| <= ulp(hi)/2.  Then
// y0 = RN(sqrt(hi/2)) lies within one ulp of sqrt(S/2), its residual
// hi/2 - y0^2 is exact under FMA, and d ~ sqrt(S/2) - y0 to within 2^-17 of
// an ulp of y0, which picks y0 or a neighbour.  The double computation lies
// within 4 * 2^-53 (relative) of sqrt(S/2), so both round to the same float
// unless sqrt(S/2) is within 2^-12 of half a spacing of a rounding midpoint
// (below a power of two the spacing halves); then, and for sums outside
// [2^-60, 2^120], it returns false and the caller takes the double path.
// About 2^-12 of the evaluations near capacity do.
template <int N>
__device__ __forceinline__ bool ref_norm_f32(const float (&f)[N], float &out)
{
    float hi = __fmul_rn(f[0], f[0]);
    float lo = __fmaf_rn(f[0], f[0], -hi);
#pragma unroll
    for (int i = 1; i < N; ++i) {
        const float ph = __fmul_rn(f[i], f[i]);
        const float pl = __fmaf_rn(f[i], f[i], -ph);
        const float sum = __fadd_rn(hi, ph);
        const float bv = __fsub_rn(sum, hi);
        const float err = __fadd_rn(__fsub_rn(hi, __fsub_rn(sum, bv)), __fsub_rn(ph, bv));
        hi = sum;
        lo = __fadd_rn(lo, __fadd_rn(pl, err));
    }
    if (!(hi >= 0x1p-60f && hi <= 0x1p120f))
        return false;
    {
        // renormalise (Fast2Sum, exact as |hi| >= |lo|)
        const float s2 = __fadd_rn(hi, lo);
        lo = __fsub_rn(lo, __fsub_rn(s2, hi));
        hi = s2;
    }
    const float h2 = __fmul_rn(hi, 0.5f);
    const float y0 = __fsqrt_rn(h2);
    const float r = __fadd_rn(__fmaf_rn(-y0, y0, h2), __fmul_rn(lo, 0.5f));
    const float d = __fmul_rn(__fmul_rn(r, 0.5f), __frcp_rn(y0));
    const int yb = __float_as_int(y0);
    const float up = __int_as_float(yb + 1);
    // half the spacing to the neighbour on d's side
    float hs = __fmul_rn(__fsub_rn(up, y0), 0.5f);
    if (d < 0.0f && (yb & 0x7fffff) == 0)
        hs = __fmul_rn(hs, 0.5f);
    const float ad = fabsf(d);
    if (fabsf(__fsub_rn(ad, hs)) <= __fmul_rn(hs, 0x1p-12f))
        return false;  // too close to a midpoint to decide in float
    out = (ad < hs) ? y0 : __int_as_float(d > 0.0f ? yb + 1 : yb - 1);
    return true;
}

// The reference's fpt from its own double computation (the undecided
// cases of ref_norm_f32).  Not inlined, so that the compiler cannot hoist its
// conversions and double additions out of the rare branch that needs them.
template <int N>
__device__ __noinline__ float ref_norm_f64(const float *f)
{
    double s = (double)f[0] * (double)f[0];
    for (int i = 1; i < N; ++i)
        s = s + (double)f[i] * (double)f[i];
    return (float)__dsqrt_rn(s * 0.5);
}

template <>
struct Proj<true> {
    // Most voxels are far inside the constraint |p| <= alpha, where the
    // reference's factor is exactly 1 (fpt <= alpha).  A float sum of the
    // squares (relative error below 7 * 2^-24) decides that case: if
    // 0.5 * s * (1 + 2^-16) < alpha^2 in float, the double |p| of the
    // reference is below alpha as well (the margin exceeds both sums'
    // rounding), so its float fpt is <= alpha and the factor is 1.  The
    // other voxels -- the flow at or near its capacity -- get the
    // reference's float fpt from ref_norm_f32, or in the rare undecidable
    // cases from the reference's own double computation: the same bits as
    // the reference, mostly at FP32 cost.
    __device__ __forceinline__ static bool surely_inside(float s, float alpha)
    {
        const float lhs = __fmul_rn(__fmul_rn(s, 0.5f), 1.0f + 0x1p-16f);
        return lhs < __fmul_rn(alpha, alpha);
    }
    template <int N>
    __device__ __forceinline__ static float factor(const float (&f)[N], float alpha)
    {
        float sf = __fmul_rn(f[0], f[0]);
#pragma unroll
        for (int i = 1; i < N; ++i)
            sf = __fmaf_rn(f[i], f[i], sf);
        // All faces zero: fpt = 0 is not above alpha >= 0, so the factor is 1.
        // This is also every cell outside the volume (zero flows and zero
        // alpha from the tile loads' out-of-range fill).
        if (sf == 0.0f && alpha >= 0.0f)
            return 1.0f;
        if (surely_inside(sf, alpha))
            return 1.0f;
        float fpt;
        if (!ref_norm_f32<N>(f, fpt))
            fpt = ref_norm_f64<N>(f);
        return finish(fpt, alpha);
    }
    // faces in the reference's summation order
    __device__ __forceinline__ static float gk(float f0, float f1, float f2, float f3, float alpha)
    {
        const float f[4] = {f0, f1, f2, f3};
        return factor<4>(f, alpha);
    }
    __device__ __forceinline__ static float gk(float f0, float f1, float f2, float f3, float f4,
                                               float f5, float alpha)
    {
        const float f[6] = {f0, f1, f2, f3, f4, f5};
        return factor<6>(f, alpha);
    }
    // fpt -> 1 / (fpt / alpha) when fpt > alpha, else 1, in float as the
    // reference (maxflow/asetsBinaryMF3D_mex.c:317-331)
    __device__ __forceinline__ static float finish(float fpt, float alpha)
    {
        fpt = (fpt > alpha) ? __fdiv_rn(fpt, alpha) : 1.0f;
        return __fdiv_rn(1.0f, fpt);
    }
};

template <>
struct Proj<false> {
    __device__ __forceinline__ static float gk(float f0, float f1, float f2, float f3, float alpha)
    {
        float s = __fmul_rn(f0, f0);
        s = __fmaf_rn(f1, f1, s);
        s = __fmaf_rn(f2, f2, s);
        s = __fmaf_rn(f3, f3, s);
        return finish(s, alpha);
    }
    __device__ __forceinline__ static float gk(float f0, float f1, float f2, float f3, float f4,
                                               float f5, float alpha)
    {
        float s = __fmul_rn(f0, f0);
        s = __fmaf_rn(f1, f1, s);
        s = __fmaf_rn(f2, f2, s);
        s = __fmaf_rn(f3, f3, s);
        s = __fmaf_rn(f4, f4, s);
        s = __fmaf_rn(f5, f5, s);
        return finish(s, alpha);
    }
    __device__ __forceinline__ static float finish(float s, float alpha)
    {
        // min(1, alpha/|p|) from the hardware reciprocal square root: equal
        // to the reference's (|p| > alpha ? 1/(|p|/alpha) : 1) up to a few
        // roundings (|p| = 0 gives alpha*inf = inf, so 1).
        return fminf(1.0f, alpha * rsqrtf(s * 0.5f));
    }
};

// x / d rounded to nearest for a fixed divisor, given rd = RN(1/d).
// Markstein's correction (Markstein, "Computation of elementary functions on
// the IBM RISC System/6000", 1990): with q = RN(x*rd) within one ulp of x/d,
// the residual x - q*d is exact under FMA and q + residual*rd rounds to
// RN(x/d).  It needs every intermediate in the normal range, so x outside
// [2^-100, 2^100] in magnitude (zero, tiny, huge, non-finite) takes the IEEE
// division.  tests/test_gpu_kernels.py compares it with __fdiv_rn over all
// 2^32 inputs for several divisors.
__device__ __forceinline__ float div_by(float x, float d, float rd)
{
    const float ax = fabsf(x);
    if (ax == 0.0f)
        return __fmul_rn(x, rd);  // +-0: the IEEE quotient keeps the sign
    if (ax >= 0x1p-100f && ax <= 0x1p100f) {
        const float q = __fmul_rn(x, rd);
        const float r = __fmaf_rn(-q, d, x);
        return __fmaf_rn(r, rd, q);
    }
    return __fdiv_rn(x, d);
}

// u/cc: EXACT takes the correctly rounded quotient (the reference's float
// division); the fast path multiplies by the rounded reciprocal (within one
// ulp of it).
template <bool EXACT>
__device__ __forceinline__ float div_cc(float x, float cc, float inv_cc)
{
    if constexpr (EXACT)
        return div_by(x, cc, inv_cc);
    else
        return x * inv_cc;
}

// MIN of the reference macros: `a < b ? a : b` (NaN picks b).
__device__ __forceinline__ float min_ref(float a, float b) { return (a < b) ? a : b; }
// ABS of the reference macros; identical to fabsf except for the sign of a NaN.
__device__ __forceinline__ float abs_ref(float x) { return fabsf(x); }

// EXACT keeps the reference's select and MIN forms; the fast path zeroes a
// border term by multiplying with a 0/1 mask (FMA pipe instead of the
// half-rate ALU pipe) and takes the hardware min.
template <bool EXACT>
__device__ __forceinline__ float keep_if(float v, bool ok, float okf)
{
    if constexpr (EXACT)
        return ok ? v : 0.0f;
    else
        return v * okf;
}
template <bool EXACT>
__device__ __forceinline__ float min_sel(float a, float b)
{
    if constexpr (EXACT)
        return min_ref(a, b);
    else
        return fminf(a, b);
}

// The cold binary start's state (stencil3d_kernel.cuh): from the reference's
// initial state on, a cell has u > 0 only where pt = Ct, so one float v holds
// both: pt itself where u = 0, else u scaled by 2^112, told apart by the
// magnitude.  Both keep all their bits.  Costs and capacities are below 2^34
// (kColdInputLimit), so that pt, at least Cs less a divergence of at most 8.5
// capacities, stays below 2^44 in magnitude, and u, at most 1 and a few roundings
// of such values times cc <= 1, below 2^14; only a u below 2^-68 counts as 0.
constexpr float kColdScale = 0x1p112f, kColdUnscale = 0x1p-112f, kColdSplit = 0x1p44f;

__device__ __forceinline__ float cold_u(float v)
{
    return fabsf(v) >= kColdSplit ? v * kColdUnscale : 0.0f;
}
__device__ __forceinline__ float cold_pt(float v, float ct) { return fabsf(v) >= kColdSplit ? ct : v; }
// v of a new pt and u; sets u to the value that v holds
__device__ __forceinline__ float cold_v(float pt, float ct, float &u)
{
    const bool sat = (pt == ct) && (u >= kColdSplit * kColdUnscale);
    u = sat ? fminf(u, 0x1p14f) : 0.0f;
    return sat ? u * kColdScale : pt;
}

// Programmatic dependent launch: lets the next launch of the stream begin
// (those made so) / waits until the launches before have finished and their
// writes are visible (returns at once where there are none).
__device__ __forceinline__ void grid_launch_dependents()
{
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
__device__ __forceinline__ void grid_dependency_wait()
{
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

// A sum of floats as an unevaluated pair (TwoSum, Knuth): about 48 bits, at
// float speed.
struct FloatPair {
    float hi = 0.f, lo = 0.f;
    __device__ __forceinline__ void add(float x, float x_lo = 0.f)
    {
        const float s = __fadd_rn(hi, x), bv = __fsub_rn(s, hi);
        const float e = __fadd_rn(__fsub_rn(hi, __fsub_rn(s, bv)), __fsub_rn(x, bv));
        lo = __fadd_rn(__fadd_rn(lo, x_lo), e);
        hi = s;
    }
    // infinities and NaN as the sum of doubles has them
    __device__ __forceinline__ double value() const { return isfinite(hi) ? (double)hi + (double)lo : (double)hi; }
};

// Sum of a per-thread value over the block (in a fixed order), valid in thread
// 0.  In pairs: the FP64 pipe takes 16 cycles for a warp's addition, so that
// the same sum in double took 3,000 to 4,500 cycles of a block of sixteen
// warps at the end of each iteration (700 here).
template <int NT>
__device__ __forceinline__ double block_sum(FloatPair v, double *scratch)
{
    static_assert(NT <= 1024, "one pair of each warp to the second step's lanes");
    auto warp_sum = [&]() {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float hi = __shfl_xor_sync(0xffffffffu, v.hi, o), lo = __shfl_xor_sync(0xffffffffu, v.lo, o);
            v.add(hi, lo);
        }
    };
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    float2 *pairs = reinterpret_cast<float2 *>(scratch);
    warp_sum();
    if (lane == 0)
        pairs[warp] = make_float2(v.hi, v.lo);
    __syncthreads();
    if (warp == 0) {
        const float2 p = lane < NT / 32 ? pairs[lane] : make_float2(0.f, 0.f);
        v.hi = p.x;
        v.lo = p.y;
        warp_sum();
    }
    return v.value();
}
template <int NT>
__device__ __forceinline__ double block_sum(float v, double *scratch)
{
    FloatPair p;
    p.hi = v;
    return block_sum<NT>(p, scratch);
}

// A lane's share of n partial sums written by other blocks: p[lane], p[lane +
// 32], ... added in order, eight loads in flight (in a loop that ends within
// the eight, a load each 600 cycles).
__device__ __forceinline__ double lane_partials(const double *p, int n, int stride = 1)
{
    double acc = 0.0;
    for (int b0 = threadIdx.x & 31; b0 < n; b0 += 256) {
        double v[8];
#pragma unroll
        for (int k = 0; k < 8; ++k)
            v[k] = b0 + 32 * k < n ? __ldcg(p + (size_t)(b0 + 32 * k) * stride) : 0.0;
#pragma unroll
        for (int k = 0; k < 8; ++k)
            acc += v[k];
    }
    return acc;
}

}  // namespace asets
