// The 3D solvers' carried state outside the iteration kernels
// (stencil3d_kernel.cuh): the gradient source gk of an initial state, and
// the source/sink flows that the iteration does not store, formed on request
// from the state before the last iteration.
//
// Streaming passes, one warp per row (rows are contiguous along r).  Built
// without contraction, so the EXACT forms are the reference's expressions.
#include "device_common.cuh"
#include "internal.h"

namespace asets {

constexpr int kCarryThreads = 256;

// divergence at element o (row r, column c, plane s) of the lower-face flows,
// in the reference's order (row, column, stream); the faces past the upper
// border are zero
__device__ __forceinline__ float div_at(const CarryArgs &A, long long o, int r, int c, int s)
{
    float d = (r + 1 < A.g.nr ? A.br[o + 1] : 0.f) - A.br[o];
    d = d + (c + 1 < A.g.nc ? A.bc[o + A.g.pitch] : 0.f);
    d = d - A.bc[o];
    d = d + (s + 1 < A.g.ns ? A.bs[o + A.g.plane] : 0.f);
    return d - A.bs[o];
}

// gk = div b - ((s0 - s1) + u/cc) of the initial state; br == null: zero flows
template <int MODEL, bool EXACT>
__global__ void __launch_bounds__(kCarryThreads) source_kernel(const CarryArgs A)
{
    const int lane = threadIdx.x & 31;
    const long long per = (long long)A.g.nc * A.g.ns, rows = per * A.flow_labels;
    const long long step = (long long)gridDim.x * (kCarryThreads / 32);
    for (long long q = blockIdx.x * (long long)(kCarryThreads / 32) + (threadIdx.x >> 5); q < rows;
         q += step) {
        const long long v = q % per, o0 = q * A.g.pitch;
        const int c = (int)(v % A.g.nc), s = (int)(v / A.g.nc);
        for (int r = lane; r < A.g.nr; r += 32) {
            const long long o = o0 + r;
            const float d = A.br ? div_at(A, o, r, c, s) : 0.f;
            float s0, s1;
            if (MODEL == 2) {
                s0 = A.pt[o];
                s1 = A.pt[o + A.g.cells];
            } else {
                s0 = A.ps[MODEL == 1 ? v * A.g.pitch + r : o];
                s1 = A.pt[o];
            }
            A.gk[o] = d - ((s0 - s1) + div_cc<EXACT>(A.u[o], A.cc, A.inv_cc));
        }
    }
}

// u or pt of the cold start's state v
__global__ void __launch_bounds__(kCarryThreads) cold_state_kernel(const CarryArgs A)
{
    const int lane = threadIdx.x & 31;
    const long long rows = (long long)A.g.nc * A.g.ns;
    const long long step = (long long)gridDim.x * (kCarryThreads / 32);
    for (long long q = blockIdx.x * (long long)(kCarryThreads / 32) + (threadIdx.x >> 5); q < rows;
         q += step)
        for (int r = lane; r < A.g.nr; r += 32) {
            const long long o = q * A.g.pitch + r;
            if (A.u_out)
                A.u_out[o] = cold_u(A.v[o]);
            else
                A.pt_out[o] = cold_pt(A.v[o], A.ct[o]);
        }
}

// binary: ps of the last iteration from the pt and u before it (COLD: the v,
// in the place of pt) and the flows after it; Potts: pt_l from the ps and u_l
// before it and the divergence
template <int MODEL, bool EXACT, bool COLD = false>
__global__ void __launch_bounds__(kCarryThreads) flows_kernel(const CarryArgs A)
{
    const int lane = threadIdx.x & 31;
    const long long per = (long long)A.g.nc * A.g.ns, rows = per * A.flow_labels;
    const long long step = (long long)gridDim.x * (kCarryThreads / 32);
    for (long long q = blockIdx.x * (long long)(kCarryThreads / 32) + (threadIdx.x >> 5); q < rows;
         q += step) {
        const long long v = q % per, o0 = q * A.g.pitch;
        const int c = (int)(v % A.g.nc), s = (int)(v / A.g.nc);
        for (int r = lane; r < A.g.nr; r += 32) {
            const long long o = o0 + r;
            const float ucc = div_cc<EXACT>(COLD ? cold_u(A.pt[o]) : A.u[o], A.cc, A.inv_cc);
            if (MODEL == 0) {
                const float pt = COLD ? cold_pt(A.pt[o], A.ct[o]) : A.pt[o];
                const float p = ((pt - ucc) + div_at(A, o, r, c, s)) + A.inv_cc;
                A.out[o] = min_sel<EXACT>(p, A.cs[o]);
            } else {
                const float p = (A.ps[v * A.g.pitch + r] + ucc) - A.dv[o];
                A.out[o] = min_ref(p, A.ct[o]);
            }
        }
    }
}

static int carry_grid(const CarryArgs &a, int num_sms)
{
    const long long rows = (long long)a.g.nc * a.g.ns * a.flow_labels;
    const long long blocks = (rows + kCarryThreads / 32 - 1) / (kCarryThreads / 32);
    const long long cap = (long long)num_sms * 8;
    return (int)(blocks < cap ? blocks : cap);
}

cudaError_t launch_source(int model, const CarryArgs &a, int num_sms, cudaStream_t st)
{
    const int grid = carry_grid(a, num_sms);
#define SRC(M)                                                     \
    if (model == M) {                                              \
        if (a.exact)                                               \
            source_kernel<M, true><<<grid, kCarryThreads, 0, st>>>(a);  \
        else                                                       \
            source_kernel<M, false><<<grid, kCarryThreads, 0, st>>>(a); \
    }
    SRC(0)
    SRC(1)
    SRC(2)
#undef SRC
    return cudaGetLastError();
}

cudaError_t launch_cold_state(const CarryArgs &a, int num_sms, cudaStream_t st)
{
    cold_state_kernel<<<carry_grid(a, num_sms), kCarryThreads, 0, st>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_flows(int model, const CarryArgs &a, int num_sms, cudaStream_t st)
{
    const int grid = carry_grid(a, num_sms);
    if (model == 0 && a.v)
        flows_kernel<0, false, true><<<grid, kCarryThreads, 0, st>>>(a);
    else if (model == 0 && a.exact)
        flows_kernel<0, true><<<grid, kCarryThreads, 0, st>>>(a);
    else if (model == 0)
        flows_kernel<0, false><<<grid, kCarryThreads, 0, st>>>(a);
    else if (a.exact)
        flows_kernel<1, true><<<grid, kCarryThreads, 0, st>>>(a);
    else
        flows_kernel<1, false><<<grid, kCarryThreads, 0, st>>>(a);
    return cudaGetLastError();
}

}  // namespace asets
