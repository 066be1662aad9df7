// Initial state of each model and the alpha(x) > 0 check.
//
//  binary:   u = (Cs - Ct >= 0), ps = pt = min(Cs, Ct)
//            (maxflow/asetsBinaryMF3D_mex.c:205-224)
//  Potts:    ps = min_l Ct, pt_l = ps, u one-hot at the FIRST argmin
//            (asetsPotts3D_mex.c:219-258)
//  Ishikawa: pt_l = min_l Ct for l < L-1 (the top layer stays 0),
//            u_l = (l < argmin) (asetsIshikawa3D_mex.c:230-270)
//
// The argmin search starts from 1e30 / 1e9 and uses `minVal > Ct` exactly
// as the reference, so ties resolve to the lowest label and a pixel whose
// costs are all >= 1e30 (or NaN) keeps the sentinel.
#include "internal.h"
#include "device_common.cuh"

namespace asets {

constexpr int kInitThreads = 256;

__device__ __forceinline__ void init_binary(const InitArgs &A, long long g)
{
    const float cs = A.cs[g], ct = A.ct[g];
    A.u[g] = (cs - ct >= 0.0f) ? 1.0f : 0.0f;
    const float m = min_ref(cs, ct);
    A.ps[g] = m;
    A.pt[g] = m;
}

__device__ __forceinline__ void argmin_labels(const float *ct, long long g, long long S, int L,
                                              float &mv, int &mi)
{
    mv = 1e30f;
    mi = 1000000000;
    for (int l = 0; l < L; ++l) {
        const float v = ct[g + l * S];
        if (mv > v) {
            mv = v;
            mi = l;
        }
    }
}

__device__ __forceinline__ void init_potts(const InitArgs &A, long long g)
{
    const long long S = A.label_stride;
    float mv;
    int mi;
    argmin_labels(A.ct, g, S, A.nlab, mv, mi);
    A.ps[g] = mv;
    for (int l = 0; l < A.nlab; ++l) {
        A.pt[g + l * S] = mv;
        A.u[g + l * S] = (l == mi) ? 1.0f : 0.0f;
    }
}

__device__ __forceinline__ void init_ishikawa(const InitArgs &A, long long g)
{
    const long long S = A.label_stride;
    float mv;
    int mi;
    argmin_labels(A.ct, g, S, A.nlab, mv, mi);
    for (int l = 0; l < A.nlab - 1; ++l) {
        A.pt[g + l * S] = mv;
        A.u[g + l * S] = (l >= mi) ? 0.0f : 1.0f;
    }
    A.pt[g + (A.nlab - 1) * S] = 0.0f;
}

// MODEL 0-2: the model's state (binary: with gk not null the gradient source of
// it and zero flows too); kPrepareCold: the binary state as v (cold_v) with its
// gradient source; kPrepareNone: nothing
template <int MODEL>
__device__ __forceinline__ void init_cells(const InitArgs &A, float *gk, float *v, float inv_cc)
{
    if (MODEL == kPrepareNone)
        return;
    for (long long g = blockIdx.x * (long long)kInitThreads + threadIdx.x; g < A.cells;
         g += (long long)gridDim.x * kInitThreads) {
        if ((int)((unsigned int)g % (unsigned int)A.pitch) >= A.nr)  // cells are below 2^32
            continue;
        if (MODEL == 0) {
            init_binary(A, g);
            if (gk) {  // u is 0 or 1: u/cc is u * inv_cc, rounded alike
                const float m = A.pt[g];
                gk[g] = 0.0f - ((m - m) + A.u[g] * inv_cc);
            }
        } else if (MODEL == 1) {
            init_potts(A, g);
        } else if (MODEL == 2) {
            init_ishikawa(A, g);
        } else {
            const float cs = A.cs[g], ct = A.ct[g];
            float u = (cs - ct >= 0.0f) ? 1.0f : 0.0f;
            v[g] = cold_v(min_ref(cs, ct), ct, u);
            gk[g] = 0.0f - u * inv_cc;  // zero flows, ps = pt
        }
    }
}

__global__ void init_source_kernel(const InitArgs A, float *gk, float inv_cc)
{
    init_cells<0>(A, gk, nullptr, inv_cc);
}

template <int MODEL>
__global__ void __launch_bounds__(kInitThreads) prepare_kernel(const __grid_constant__ PrepareArgs A)
{
    const long long t0 = blockIdx.x * (long long)kInitThreads + threadIdx.x;
    const long long step = (long long)gridDim.x * kInitThreads;
    if (blockIdx.x == 0) {
        // what follows the maps, which the launches have among their parameters
        const int *src = reinterpret_cast<const int *>(&A.desc);
        for (int i = sizeof(TensorMaps) / 4 + threadIdx.x; i < (int)(sizeof(ProblemDesc) / 4); i += kInitThreads)
            reinterpret_cast<int *>(A.d_desc)[i] = src[i];
        if (threadIdx.x == 0)
            *A.d_ctl = A.ctl;
        if (threadIdx.x < 4)
            A.queue[threadIdx.x] = 0;
    }
    for (long long i = t0; i < A.n_cvg; i += step)
        A.cvg[i] = 0.0f;
    for (int k = 0; k < 3; ++k)
        if (A.zero[k])
            for (long long i = t0; i < A.zero_floats / 4; i += step)
                reinterpret_cast<float4 *>(A.zero[k])[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    init_cells<MODEL>(A.init, A.gk, A.v, A.desc.inv_cc);
}

// projStep's check, `if (alpha <= 0) error` (asetsBinaryMF3D_mex.c:317-319),
// over every alpha slice the solve reads.  NaN passes, as in the reference.
__global__ void validate_alpha_kernel(InitArgs A)
{
    int bad = 0;
    const long long total = A.cells * A.alpha_labels;
    for (long long i = blockIdx.x * (long long)kInitThreads + threadIdx.x; i < total;
         i += (long long)gridDim.x * kInitThreads) {
        // label slices are whole padded volumes; elements are below 2^32
        if ((int)((unsigned int)i % (unsigned int)A.pitch) >= A.nr)
            continue;
        if (A.alpha[i] <= 0.0f)
            bad = 1;
    }
    if (__syncthreads_or(bad) && threadIdx.x == 0)
        atomicOr(&A.ctl->alpha_bad, 1);
}

__global__ void check_range_kernel(InitArgs A)
{
    int wide = 0;
    for (long long g = blockIdx.x * (long long)kInitThreads + threadIdx.x; g < A.cells;
         g += (long long)gridDim.x * kInitThreads) {
        if ((int)((unsigned int)g % (unsigned int)A.pitch) >= A.nr)
            continue;
        const float m = fmaxf(fmaxf(fabsf(A.cs[g]), fabsf(A.ct[g])), fabsf(A.alpha[g]));
        // fmaxf drops a NaN: the sum keeps it
        if (!(m < kColdInputLimit) || !(A.cs[g] + A.ct[g] + A.alpha[g] < INFINITY))
            wide = 1;
    }
    if (__syncthreads_or(wide) && threadIdx.x == 0)
        atomicOr(&A.ctl->wide, 1);
}

static int grid_for(long long n, int num_sms)
{
    long long b = (n + kInitThreads - 1) / kInitThreads;
    long long cap = (long long)num_sms * 8;
    if (b < 1)
        b = 1;
    return (int)(b < cap ? b : cap);
}

cudaError_t launch_init_source(const InitArgs &a, float *gk, float inv_cc, int num_sms, cudaStream_t st)
{
    init_source_kernel<<<grid_for(a.cells, num_sms), kInitThreads, 0, st>>>(a, gk, inv_cc);
    return cudaGetLastError();
}

cudaError_t launch_prepare(const PrepareArgs &a, int num_sms, cudaStream_t st)
{
    static_assert(sizeof(PrepareArgs) <= 4096, "kernel parameter space");
    static_assert(sizeof(ProblemDesc) % 4 == 0, "copied by words");
    const int grid = grid_for(a.init.cells, num_sms);
    switch (a.model) {
    case 0: prepare_kernel<0><<<grid, kInitThreads, 0, st>>>(a); break;
    case 1: prepare_kernel<1><<<grid, kInitThreads, 0, st>>>(a); break;
    case 2: prepare_kernel<2><<<grid, kInitThreads, 0, st>>>(a); break;
    case kPrepareCold: prepare_kernel<kPrepareCold><<<grid, kInitThreads, 0, st>>>(a); break;
    case kPrepareNone: prepare_kernel<kPrepareNone><<<grid, kInitThreads, 0, st>>>(a); break;
    default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

cudaError_t launch_validate_alpha(const InitArgs &a, int num_sms, cudaStream_t st)
{
    validate_alpha_kernel<<<grid_for(a.cells * a.alpha_labels, num_sms), kInitThreads, 0, st>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_check_range(const InitArgs &a, int num_sms, cudaStream_t st)
{
    check_range_kernel<<<grid_for(a.cells, num_sms), kInitThreads, 0, st>>>(a);
    return cudaGetLastError();
}

// Self-check of the bounded wait: one thread arms an mbarrier for 16 bytes
// of transaction that no copy will deliver and waits on it with the solver
// kernels' bounded wait, which must give up after its budget and report
// DEV_ERR_TIMEOUT.  Nothing is in flight when the kernel returns.
__global__ void wait_selftest_kernel(int *err)
{
    __shared__ uint64_t bar;
    __shared__ int abort_flag;
    if (threadIdx.x == 0) {
        abort_flag = 0;
        mbar_init(&bar, 1);
        mbar_fence_init();
        mbar_arrive_expect_tx(&bar, 16);
        if (!mbar_wait_bounded(&bar, 0, &abort_flag))
            atomicOr(err, DEV_ERR_TIMEOUT);
    }
}

cudaError_t launch_wait_selftest(int *d_err, cudaStream_t st)
{
    wait_selftest_kernel<<<1, 32, 0, st>>>(d_err);
    return cudaGetLastError();
}

}  // namespace asets
