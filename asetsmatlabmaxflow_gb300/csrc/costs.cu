// Cost terms and regularisation weights built on the GPU: the step before
// the solvers in the reference's applications (applications/*.m), as
// HBM-streaming kernels over the Matlab-layout volume.
//
//   L1 intensity      Ct_l = |I' - m_l|, I' = (I - min I)/(max I - min I)
//                     (L1IntensitySegmentation2D.m:32-45)
//   -log probability  Ct_l = -log(p_l + eps)
//                     (atlasProbabilityMapsRegularization3D.m:39-53)
//   histogram LL      Ct_l = -log10(P_l(bin(I)) + eps) from the 256-bin
//                     histogram of the voxels scribbled with label l
//                     (interactiveGraphCutSegmentation3D.m:47-49, 104-122)
//   contrast alpha    alpha = a + b*exp(-c*|grad I'|^p), central differences
//                     inside, one-sided at the border (Matlab's gradient;
//                     smoothManualSegmentations2D.m:82-91)
#include <algorithm>
#include <cmath>
#include <cstring>
#include <string>
#include <type_traits>
#include <vector>

#include "asets.h"
#include "device_common.cuh"
#include "internal.h"

using namespace asets;

namespace {

constexpr int kThreads = 256;
constexpr int kMaxLabels = 32;
constexpr int kBins = 256;

struct Labels {
    float v[kMaxLabels];
};

int grid_for(long long n, int num_sms)
{
    long long b = (n + kThreads - 1) / kThreads;
    const long long cap = (long long)num_sms * 8;
    return (int)(b < 1 ? 1 : (b < cap ? b : cap));
}

// Order-preserving map of floats to unsigned integers (for atomic min/max).
__device__ __forceinline__ unsigned int float_key(float f)
{
    const unsigned int u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__host__ __device__ inline float key_float(unsigned int k)
{
#ifdef __CUDA_ARCH__
    return __uint_as_float((k & 0x80000000u) ? (k & 0x7FFFFFFFu) : ~k);
#else
    const unsigned int u = (k & 0x80000000u) ? (k & 0x7FFFFFFFu) : ~k;
    float f;
    memcpy(&f, &u, 4);
    return f;
#endif
}

// 16-byte accesses where the arrays allow them (base 16-byte aligned; for
// label-major outputs also n % 4 == 0), so that every thread keeps several
// loads in flight; the remainder element by element.
__device__ __forceinline__ bool aligned16(const void *p)
{
    return (reinterpret_cast<uintptr_t>(p) & 15u) == 0;
}

// mm[0] = ~key(min), mm[1] = key(max), both from zero; NaNs are skipped (as
// Matlab's min/max).
__global__ void minmax_kernel(const float *x, long long n, unsigned int *mm)
{
    unsigned int lo = 0xFFFFFFFFu, hi = 0u;
    auto take = [&](float f) {
        if (f == f) {
            const unsigned int k = float_key(f);
            lo = min(lo, k);
            hi = max(hi, k);
        }
    };
    const long long t0 = blockIdx.x * (long long)kThreads + threadIdx.x;
    const long long stride = (long long)gridDim.x * kThreads;
    long long head = 0;
    if (aligned16(x)) {
        const long long n4 = n >> 2;
        const float4 *x4 = reinterpret_cast<const float4 *>(x);
#pragma unroll 4
        for (long long i = t0; i < n4; i += stride) {
            const float4 v = __ldg(x4 + i);
            take(v.x);
            take(v.y);
            take(v.z);
            take(v.w);
        }
        head = n4 << 2;
    }
    for (long long i = head + t0; i < n; i += stride)
        take(x[i]);
    // block reduction first: one atomic pair per block (same-address
    // atomics serialise in L2)
    __shared__ unsigned int s_lo[kThreads / 32], s_hi[kThreads / 32];
    for (int o = 16; o > 0; o >>= 1) {
        lo = min(lo, __shfl_xor_sync(0xffffffffu, lo, o));
        hi = max(hi, __shfl_xor_sync(0xffffffffu, hi, o));
    }
    if ((threadIdx.x & 31) == 0) {
        s_lo[threadIdx.x >> 5] = lo;
        s_hi[threadIdx.x >> 5] = hi;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < kThreads / 32; ++w) {
            lo = min(lo, s_lo[w]);
            hi = max(hi, s_hi[w]);
        }
        atomicMax(&mm[0], ~lo);
        atomicMax(&mm[1], hi);
    }
}

// (I - min) / (max - min), as Matlab's single arithmetic; the range is read
// once per thread (mm == nullptr: the identity).  The quotient is IEEE's:
// for an ordinary range by the corrected product with its reciprocal (div_by),
// three operations instead of a division's dozen.
struct Norm {
    float lo = 0.f, den = 1.f, rd = 0.f;  // rd = 0: divide
    bool on = false;
    __device__ explicit Norm(const unsigned int *mm)
    {
        if (mm) {
            lo = key_float(~mm[0]);
            den = __fsub_rn(key_float(mm[1]), lo);
            // quotients of at least 2^-100 / 2^20, all in the normal range
            if (den >= 0x1p-20f && den <= 0x1p20f)
                rd = __fdiv_rn(1.0f, den);
            on = true;
        }
    }
    __device__ float operator()(float v) const
    {
        if (!on)
            return v;
        const float x = __fsub_rn(v, lo);
        return rd != 0.f ? div_by(x, den, rd) : __fdiv_rn(x, den);
    }
};

__global__ void l1_kernel(const float *img, long long n, Labels m, int L,
                          const unsigned int *mm, float *ct)
{
    const Norm nrm(mm);
    const long long t0 = blockIdx.x * (long long)kThreads + threadIdx.x;
    const long long stride = (long long)gridDim.x * kThreads;
    long long head = 0;
    if ((n & 3) == 0 && aligned16(img) && aligned16(ct)) {
        const long long n4 = n >> 2;
        const float4 *x4 = reinterpret_cast<const float4 *>(img);
        float4 *c4 = reinterpret_cast<float4 *>(ct);
#pragma unroll 2
        for (long long i = t0; i < n4; i += stride) {
            const float4 r = __ldg(x4 + i);
            const float v0 = nrm(r.x), v1 = nrm(r.y), v2 = nrm(r.z), v3 = nrm(r.w);
            for (int l = 0; l < L; ++l) {
                const float q = m.v[l];
                __stcs(c4 + l * n4 + i, make_float4(fabsf(__fsub_rn(v0, q)), fabsf(__fsub_rn(v1, q)),
                                                    fabsf(__fsub_rn(v2, q)), fabsf(__fsub_rn(v3, q))));
            }
        }
        head = n;
    }
    for (long long i = head + t0; i < n; i += stride) {
        const float v = nrm(img[i]);
        for (int l = 0; l < L; ++l)
            ct[l * n + i] = fabsf(__fsub_rn(v, m.v[l]));
    }
}

__global__ void neglog_kernel(const float *p, long long total, float eps, float *ct)
{
    auto f = [&](float x) { return -logf(__fadd_rn(x, eps)); };
    const long long t0 = blockIdx.x * (long long)kThreads + threadIdx.x;
    const long long stride = (long long)gridDim.x * kThreads;
    long long head = 0;
    if (aligned16(p) && aligned16(ct)) {
        const long long n4 = total >> 2;
        const float4 *p4 = reinterpret_cast<const float4 *>(p);
        float4 *c4 = reinterpret_cast<float4 *>(ct);
#pragma unroll 2
        for (long long i = t0; i < n4; i += stride) {
            const float4 v = __ldg(p4 + i);
            __stcs(c4 + i, make_float4(f(v.x), f(v.y), f(v.z), f(v.w)));
        }
        head = n4 << 2;
    }
    for (long long i = head + t0; i < total; i += stride)
        ct[i] = f(p[i]);
}

// I' * 255 in single precision as computeLogLikelihoodCost forms it
__device__ __forceinline__ float scaled255(float v, const Norm &nrm)
{
    return __fmul_rn(nrm(v), 255.0f);
}

// histc(x, 0:255): bin k holds k <= x < k+1, the last bin also x == 255.
// Scribbles and image are read 16 bytes at a time, several in flight (the
// image everywhere: loads that wait for a scribble cost more than the lines
// they save).  256 x 231 x 256, one voxel in twenty scribbled: 36 us (the image
// only where scribbled: 52; one element at a time: 91).
__global__ void __launch_bounds__(kThreads) hist_kernel(const float *img, const int *scrib, long long n,
                                                        int L, const unsigned int *mm, unsigned int *hist)
{
    extern __shared__ unsigned int h[];  // L * kBins: as many blocks on an SM as threads allow
    const Norm nrm(mm);
    for (int i = threadIdx.x; i < L * kBins; i += kThreads)
        h[i] = 0;
    __syncthreads();
    auto take = [&](int lab, float v) {
        if (lab < 1 || lab > L)
            return;
        const float x = scaled255(v, nrm);
        if (!(x >= 0.f && x <= 255.f))
            return;
        const int b = min((int)floorf(x), kBins - 1);
        atomicAdd(&h[(lab - 1) * kBins + b], 1u);
    };
    const long long t0 = blockIdx.x * (long long)kThreads + threadIdx.x;
    const long long stride = (long long)gridDim.x * kThreads;
    long long head = 0;
    if (aligned16(scrib) && aligned16(img)) {
        const long long n4 = n >> 2;
        const int4 *s4 = reinterpret_cast<const int4 *>(scrib);
        const float4 *x4 = reinterpret_cast<const float4 *>(img);
        constexpr int kAhead = 4;
        for (long long i = t0; i < n4; i += kAhead * stride) {
            int4 v[kAhead];
            float4 x[kAhead];
#pragma unroll
            for (int j = 0; j < kAhead; ++j) {
                const bool ok = i + j * stride < n4;
                v[j] = ok ? __ldcs(s4 + i + j * stride) : make_int4(0, 0, 0, 0);
                x[j] = ok ? __ldg(x4 + i + j * stride) : make_float4(0.f, 0.f, 0.f, 0.f);
            }
#pragma unroll
            for (int j = 0; j < kAhead; ++j) {
                take(v[j].x, x[j].x);
                take(v[j].y, x[j].y);
                take(v[j].z, x[j].z);
                take(v[j].w, x[j].w);
            }
        }
        head = n4 << 2;
    }
    for (long long i = head + t0; i < n; i += stride)
        take(scrib[i], img[i]);
    __syncthreads();
    for (int i = threadIdx.x; i < L * kBins; i += kThreads)
        if (h[i])
            atomicAdd(&hist[i], h[i]);
}

// Per-bin cost of label blockIdx.x in double, as the reference's
// binCounts./sum and -log10(P + epsilon), rounded to float (NaN if no scribble).
__global__ void __launch_bounds__(kBins) cost_table_kernel(const unsigned int *hist, double eps, float *table)
{
    __shared__ unsigned long long s_sum[kBins / 32];
    const int i = blockIdx.x * kBins + threadIdx.x;
    const unsigned int h = hist[i];
    unsigned long long t = h;
    for (int o = 16; o > 0; o >>= 1)
        t += __shfl_xor_sync(0xffffffffu, t, o);
    if ((threadIdx.x & 31) == 0)
        s_sum[threadIdx.x >> 5] = t;
    __syncthreads();
    unsigned long long total = 0;
    for (int w = 0; w < kBins / 32; ++w)
        total += s_sum[w];
    table[i] = (float)(-log10((double)h / (double)total + eps));
}

// Ct_l = cost_l[uint16(I'*255)]: Matlab's uint16() rounds half away from zero.
__global__ void lookup_kernel(const float *img, long long n, int L, const unsigned int *mm,
                              const float *table, float *ct)
{
    const Norm nrm(mm);
    auto bin = [&](float v) {
        const int b = (int)roundf(scaled255(v, nrm));
        return b < 0 ? 0 : (b > kBins - 1 ? kBins - 1 : b);
    };
    const long long t0 = blockIdx.x * (long long)kThreads + threadIdx.x;
    const long long stride = (long long)gridDim.x * kThreads;
    long long head = 0;
    if ((n & 3) == 0 && aligned16(img) && aligned16(ct)) {
        const long long n4 = n >> 2;
        const float4 *x4 = reinterpret_cast<const float4 *>(img);
        float4 *c4 = reinterpret_cast<float4 *>(ct);
        for (long long i = t0; i < n4; i += stride) {
            const float4 v = __ldg(x4 + i);
            const int b0 = bin(v.x), b1 = bin(v.y), b2 = bin(v.z), b3 = bin(v.w);
            for (int l = 0; l < L; ++l) {
                const float *t = table + l * kBins;
                __stcs(c4 + l * n4 + i, make_float4(t[b0], t[b1], t[b2], t[b3]));
            }
        }
        head = n;
    }
    for (long long i = head + t0; i < n; i += stride) {
        const int b = bin(img[i]);
        for (int l = 0; l < L; ++l)
            ct[l * n + i] = table[l * kBins + b];
    }
}

// alpha = a + b*exp(-c*|grad I'|^p) (p = 1 or 2), replicated over L slices.
// Matlab's gradient: (f(k+1) - f(k-1))/2 inside, one-sided at the ends, 0 on an
// axis of length 1.  The differences are taken of the image itself and scaled
// by 1/(max - min) after: closer to the exact gradient than differences of
// rounded quotients, and no division per voxel.
//
// A thread owns VEC (4 or 1) adjacent rows of one column and walks some planes,
// with the planes z-1, z, z+1 in registers; the rows beside come from the
// neighbouring lanes, the columns beside from L1 and L2.  16-byte accesses
// (VEC = 4) where rows are whole multiples of them.  256 x 231 x 256: 52
// us for one label, 67 for four, which the stores bound (a 32 x 8 tile in
// shared memory, every voxel normalised: 138 and 152).
constexpr int kAWarps = 8, kAZ = 16;  // columns and planes of a block

template <int VEC>
struct Rows {
    float v[VEC];
};

template <int VEC>
__device__ __forceinline__ Rows<VEC> ld_rows(const float *p, bool ok)
{
    Rows<VEC> r;
    if constexpr (VEC == 4) {
        const float4 t = ok ? __ldg(reinterpret_cast<const float4 *>(p)) : make_float4(0.f, 0.f, 0.f, 0.f);
        r.v[0] = t.x;
        r.v[1] = t.y;
        r.v[2] = t.z;
        r.v[3] = t.w;
    } else {
        r.v[0] = ok ? __ldg(p) : 0.f;
    }
    return r;
}

template <int VEC>
__global__ void __launch_bounds__(32 * kAWarps)
    alpha_kernel(const float *img, int ny, int nx, int nz, const unsigned int *mm, float a, float b, float c,
                 int squared, int L, int az, int per, float *alpha)
{
    // `per` lanes have a column's rows; short columns share a warp
    const int lane = threadIdx.x & 31, share = 32 / per, col = lane / per;
    const int y = (blockIdx.x * per + lane - col * per) * VEC;
    const int x0 = (blockIdx.y * kAWarps + (threadIdx.x >> 5)) * share, x = x0 + col;
    if (x0 >= nx)
        return;  // a whole warp
    const int z0 = blockIdx.z * az, z1 = min(nz, z0 + az);
    const bool in = y < ny && x < nx && col < share;
    const long long plane = (long long)ny * nx, n = plane * nz;
    const float *p = img + (long long)x * ny + y;
    // 1/(max - min); a range whose reciprocal is not an ordinary number (and
    // one that is not finite, or zero) takes the quotients themselves
    float low = 0.f, den = 1.f, rd = 1.f;
    if (mm) {
        low = key_float(~mm[0]);
        den = __fsub_rn(key_float(mm[1]), low);
        rd = __fdiv_rn(1.f, den);
    }
    const bool plain = !mm || (fabsf(low) < INFINITY && den >= 0x1p-100f && den <= 0x1p100f);
    auto unit = [&](float hi, float lo, float half) {
        if (plain)
            return __fmul_rn(__fmul_rn(__fsub_rn(hi, lo), half), rd);
        return __fmul_rn(__fsub_rn(__fdiv_rn(__fsub_rn(hi, low), den), __fdiv_rn(__fsub_rn(lo, low), den)), half);
    };
    const bool x_lo = x > 0, x_up = x + 1 < nx;
    const float sx = (x_lo && x_up) ? 0.5f : 1.f;
    // the rows beyond the warp's 32*VEC (a shared warp's columns are whole)
    const bool edge_lo = lane == 0 && in && y > 0, edge_up = lane == 31 && in && y + VEC < ny;
    const long long z_off = (long long)z0 * plane;
    Rows<VEC> cur = ld_rows<VEC>(p + z_off, in), lo = z0 > 0 ? ld_rows<VEC>(p + z_off - plane, in) : cur;
    for (int z = z0; z < z1; ++z) {
        const float *q = p + (long long)z * plane;
        const Rows<VEC> up = z + 1 < nz ? ld_rows<VEC>(q + plane, in) : cur;
        const Rows<VEC> xl = x_lo ? ld_rows<VEC>(q - ny, in) : cur;
        const Rows<VEC> xu = x_up ? ld_rows<VEC>(q + ny, in) : cur;
        float yl = __shfl_up_sync(0xffffffffu, cur.v[VEC - 1], 1);
        float yu = __shfl_down_sync(0xffffffffu, cur.v[0], 1);
        if (edge_lo)
            yl = __ldg(q - 1);
        if (edge_up)
            yu = __ldg(q + VEC);
        const float sz = (z > 0 && z + 1 < nz) ? 0.5f : 1.f;
        float al[VEC];
#pragma unroll
        for (int j = 0; j < VEC; ++j) {
            const int yy = y + j;
            const bool y_lo = yy > 0, y_up = yy + 1 < ny;
            const float vl = y_lo ? (j ? cur.v[j - 1] : yl) : cur.v[j];
            const float vu = y_up ? (j + 1 < VEC ? cur.v[j + 1 < VEC ? j + 1 : j] : yu) : cur.v[j];
            // an axis of length 1 adds nothing, whatever the value there
            const float gy = ny < 2 ? 0.f : unit(vu, vl, (y_lo && y_up) ? 0.5f : 1.f);
            const float gx = nx < 2 ? 0.f : unit(xu.v[j], xl.v[j], sx);
            float g2 = __fmaf_rn(gx, gx, __fmul_rn(gy, gy));
            if (nz > 1) {
                const float gz = unit(up.v[j], lo.v[j], sz);
                g2 = __fmaf_rn(gz, gz, g2);
            }
            const float t = squared ? g2 : __fsqrt_rn(g2);
            al[j] = __fadd_rn(a, __fmul_rn(b, expf(__fmul_rn(-c, t))));
        }
        if (in) {
            float *o = alpha + (long long)z * plane + (long long)x * ny + y;
            for (int l = 0; l < L; ++l) {
                if constexpr (VEC == 4)
                    __stcs(reinterpret_cast<float4 *>(o + l * n), make_float4(al[0], al[1], al[2], al[3]));
                else
                    __stcs(o + l * n, al[0]);
            }
        }
        lo = cur;
        cur = up;
    }
}

struct Scratch {
    std::vector<void *> ptrs;
    cudaStream_t st;
    cudaMemPool_t pool;
    explicit Scratch(asets_context *ctx) : st(context_stream(ctx)), pool(context_pool(ctx)) {}
    template <class T>
    cudaError_t get(T **p, size_t bytes)
    {
        void *v = nullptr;
        const size_t b = bytes < 4 ? 4 : bytes;
        cudaError_t e = pool ? cudaMallocFromPoolAsync(&v, b, pool, st) : cudaMallocAsync(&v, b, st);
        if (e == cudaSuccess)
            ptrs.push_back(v);
        *p = static_cast<T *>(v);
        return e;
    }
    ~Scratch()
    {
        for (void *p : ptrs)
            cudaFreeAsync(p, st);
        cudaStreamSynchronize(st);
    }
};

#define CT_TRY(call)                                                                       \
    do {                                                                                   \
        cudaError_t e_ = (call);                                                           \
        if (e_ != cudaSuccess) {                                                           \
            cudaGetLastError();                                                            \
            set_last_error((std::string(#call) + ": " + cudaGetErrorString(e_)).c_str()); \
            return e_ == cudaErrorMemoryAllocation ? ASETS_ERR_OUT_OF_MEMORY : ASETS_ERR_CUDA; \
        }                                                                                  \
    } while (0)

// A device view of a caller array: the array itself, or a device copy of a
// host array (copied back on `finish` for outputs).
template <class T>
struct View {
    T *d = nullptr;
    const T *host_in = nullptr;
    T *host_out = nullptr;
    size_t count = 0;
};

template <class T>
cudaError_t in_view(Scratch &s, asets_memory where, const T *p, size_t count, View<T> &v)
{
    v.count = count;
    if (where == ASETS_DEVICE) {
        v.d = const_cast<T *>(p);
        return cudaSuccess;
    }
    cudaError_t e = s.get(&v.d, count * sizeof(T));
    if (e != cudaSuccess)
        return e;
    return cudaMemcpyAsync(v.d, p, count * sizeof(T), cudaMemcpyHostToDevice, s.st);
}

template <class T>
cudaError_t out_view(Scratch &s, asets_memory where, T *p, size_t count, View<T> &v)
{
    v.count = count;
    if (where == ASETS_DEVICE) {
        v.d = p;
        return cudaSuccess;
    }
    v.host_out = p;
    return s.get(&v.d, count * sizeof(T));
}

template <class T>
cudaError_t finish(Scratch &s, View<T> &v)
{
    if (v.host_out)
        return cudaMemcpyAsync(v.host_out, v.d, v.count * sizeof(T), cudaMemcpyDeviceToHost, s.st);
    return cudaSuccess;
}

// Scratch words of a call, set to zero: the range (two words) first.
cudaError_t zeroed(Scratch &s, size_t words, unsigned int **p)
{
    cudaError_t e = s.get(p, words * sizeof(unsigned int));
    return e == cudaSuccess ? cudaMemsetAsync(*p, 0, words * sizeof(unsigned int), s.st) : e;
}

cudaError_t run_minmax(Scratch &s, const float *x, long long n, int sms, unsigned int *mm)
{
    minmax_kernel<<<grid_for(n, sms), kThreads, 0, s.st>>>(x, n, mm);
    return cudaGetLastError();
}

struct CtxUse {
    int prev = 0;
    explicit CtxUse(asets_context *ctx)
    {
        cudaGetDevice(&prev);
        cudaSetDevice(context_device(ctx));
    }
    ~CtxUse() { cudaSetDevice(prev); }
};

}  // namespace

extern "C" ASETS_API asets_status asets_cost_l1(asets_context *ctx, asets_memory where,
                                                const float *img, long long n,
                                                const float *models, int L, int normalize,
                                                float *Ct)
{
    if (!ctx || !img || !models || !Ct || n < 1 || L < 1 || L > kMaxLabels) {
        set_last_error("asets_cost_l1: bad arguments (1 <= L <= 32)");
        return ASETS_ERR_INVALID_ARG;
    }
    CtxUse use(ctx);
    Scratch s(ctx);
    View<float> vi, vo;
    CT_TRY(in_view(s, where, img, (size_t)n, vi));
    CT_TRY(out_view(s, where, Ct, (size_t)n * L, vo));
    unsigned int *mm = nullptr;
    if (normalize) {
        CT_TRY(zeroed(s, 2, &mm));
        CT_TRY(run_minmax(s, vi.d, n, context_num_sms(ctx), mm));
    }
    Labels m{};
    for (int l = 0; l < L; ++l)
        m.v[l] = models[l];
    l1_kernel<<<grid_for(n, context_num_sms(ctx)), kThreads, 0, s.st>>>(vi.d, n, m, L, mm, vo.d);
    CT_TRY(cudaGetLastError());
    CT_TRY(finish(s, vo));
    CT_TRY(cudaStreamSynchronize(s.st));
    return ASETS_OK;
}

extern "C" ASETS_API asets_status asets_cost_neglog(asets_context *ctx, asets_memory where,
                                                    const float *prob, long long n, int L,
                                                    float eps, float *Ct)
{
    if (!ctx || !prob || !Ct || n < 1 || L < 1) {
        set_last_error("asets_cost_neglog: bad arguments");
        return ASETS_ERR_INVALID_ARG;
    }
    CtxUse use(ctx);
    Scratch s(ctx);
    View<float> vi, vo;
    const long long total = n * L;
    CT_TRY(in_view(s, where, prob, (size_t)total, vi));
    CT_TRY(out_view(s, where, Ct, (size_t)total, vo));
    neglog_kernel<<<grid_for(total, context_num_sms(ctx)), kThreads, 0, s.st>>>(vi.d, total, eps,
                                                                               vo.d);
    CT_TRY(cudaGetLastError());
    CT_TRY(finish(s, vo));
    CT_TRY(cudaStreamSynchronize(s.st));
    return ASETS_OK;
}

extern "C" ASETS_API asets_status asets_cost_histogram_ll(asets_context *ctx, asets_memory where,
                                                          const float *img, const int *scribbles,
                                                          long long n, int L, double eps,
                                                          float *Ct, unsigned int *hist_out)
{
    if (!ctx || !img || !scribbles || !Ct || n < 1 || L < 1 || L > kMaxLabels) {
        set_last_error("asets_cost_histogram_ll: bad arguments (1 <= L <= 32)");
        return ASETS_ERR_INVALID_ARG;
    }
    CtxUse use(ctx);
    const int sms = context_num_sms(ctx);
    Scratch s(ctx);
    View<float> vi, vo;
    View<int> vs;
    CT_TRY(in_view(s, where, img, (size_t)n, vi));
    CT_TRY(in_view(s, where, scribbles, (size_t)n, vs));
    CT_TRY(out_view(s, where, Ct, (size_t)n * L, vo));
    // the range, the counts and (written whole) the table
    const size_t bins = (size_t)L * kBins;
    unsigned int *mm = nullptr;
    CT_TRY(zeroed(s, 2 + 2 * bins, &mm));
    unsigned int *hist = mm + 2;
    float *table = reinterpret_cast<float *>(hist + bins);
    CT_TRY(run_minmax(s, vi.d, n, sms, mm));
    hist_kernel<<<grid_for(n, sms), kThreads, bins * sizeof(unsigned int), s.st>>>(vi.d, vs.d, n, L, mm, hist);
    CT_TRY(cudaGetLastError());
    cost_table_kernel<<<L, kBins, 0, s.st>>>(hist, eps, table);
    CT_TRY(cudaGetLastError());
    lookup_kernel<<<grid_for(n, sms), kThreads, 0, s.st>>>(vi.d, n, L, mm, table, vo.d);
    CT_TRY(cudaGetLastError());
    CT_TRY(finish(s, vo));
    if (hist_out)
        CT_TRY(cudaMemcpyAsync(hist_out, hist, bins * sizeof(unsigned int),
                               cudaMemcpyDeviceToHost, s.st));
    CT_TRY(cudaStreamSynchronize(s.st));
    return ASETS_OK;
}

extern "C" ASETS_API asets_status asets_alpha_contrast(asets_context *ctx, asets_memory where,
                                                       const float *img, int Ny, int Nx, int Nz,
                                                       int normalize, float a, float b, float c,
                                                       int squared, int L, float *alpha)
{
    if (!ctx || !img || !alpha || Ny < 1 || Nx < 1 || Nz < 1 || L < 1 ||
        (Nx - 1) / kAWarps > 65534 || (Nz - 1) / 32 > 65534) {
        set_last_error("asets_alpha_contrast: bad arguments");
        return ASETS_ERR_INVALID_ARG;
    }
    CtxUse use(ctx);
    const int sms = context_num_sms(ctx);
    const long long n = (long long)Ny * Nx * Nz;
    Scratch s(ctx);
    View<float> vi, vo;
    CT_TRY(in_view(s, where, img, (size_t)n, vi));
    CT_TRY(out_view(s, where, alpha, (size_t)n * L, vo));
    unsigned int *mm = nullptr;
    if (normalize) {
        CT_TRY(zeroed(s, 2, &mm));
        CT_TRY(run_minmax(s, vi.d, n, sms, mm));
    }
    const int az = std::max(kAZ, (Nz + 65534) / 65535);  // planes per block: the grid's z extent
    auto launch = [&](auto vec) {
        constexpr int V = decltype(vec)::value;
        const int lanes = (Ny + V - 1) / V, per = lanes <= 16 ? lanes : 32, cols = kAWarps * (32 / per);
        const dim3 grid((lanes + per - 1) / per, (Nx + cols - 1) / cols, (Nz + az - 1) / az);
        alpha_kernel<V><<<grid, 32 * kAWarps, 0, s.st>>>(vi.d, Ny, Nx, Nz, mm, a, b, c, squared, L, az, per, vo.d);
    };
    const bool vec4 = (Ny & 3) == 0 && ((reinterpret_cast<uintptr_t>(vi.d) | reinterpret_cast<uintptr_t>(vo.d)) & 15) == 0;
    if (vec4)
        launch(std::integral_constant<int, 4>{});
    else
        launch(std::integral_constant<int, 1>{});
    CT_TRY(cudaGetLastError());
    CT_TRY(finish(s, vo));
    CT_TRY(cudaStreamSynchronize(s.st));
    return ASETS_OK;
}
