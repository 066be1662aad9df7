// Test helper: the five-layer weight-gradient launch on positive operands (so
// that roundings of one sign show) against sums in double, half-planar layout.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cmath>
#include <cstdint>
#include <cstring>
#include <vector>

#include "wgrad_tc.cuh"

// values in [0.5, 1), zero in the rows' padding
__global__ void fill_kernel(__nv_bfloat16 *p, int ny, long long rows, unsigned int seed)
{
    const long long yp = (ny + 7) / 8 * 8, n = yp * rows * 16;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x) {
        unsigned int z = (unsigned int)i * 2654435761u + seed;
        z = (z ^ (z >> 15)) * 2246822519u;
        z ^= z >> 13;
        p[i] = __float2bfloat16_rn((i / 8) % yp < ny ? 0.5f + (float)(z >> 9) * 0x1p-24f : 0.f);
    }
}

// the middle tap of channel pair (ci, co): the products of the same voxels
__global__ void ref_kernel(const __nv_bfloat16 *a, const __nv_bfloat16 *g, int ny, long long rows, double *sum)
{
    const int ci = blockIdx.x / 16, co = blockIdx.x % 16;
    const long long yp = (ny + 7) / 8 * 8;
    double s = 0.0;
    for (long long v = threadIdx.x; v < yp * rows; v += blockDim.x) {
        const long long r = v / yp, y = v % yp;
        s += (double)__bfloat162float(a[(r * 2 + ci / 8) * yp * 8 + y * 8 + ci % 8]) *
             (double)__bfloat162float(g[(r * 2 + co / 8) * yp * 8 + y * 8 + co % 8]);
    }
    atomicAdd(&sum[blockIdx.x], s);
}

// Returns 0 and the largest relative error over the five layers.
extern "C" __attribute__((visibility("default"))) int wgrad_layers_check(int ny, int nx, int nz, double *worst_out)
{
    void *fn = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &fn, 12000, cudaEnableDefault, &q) !=
            cudaSuccess || !fn)
        return 1;
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const long long rows = (long long)nx * nz, elems = (long long)((ny + 7) / 8 * 8) * rows * 16;
    constexpr int kOut = 27 * 256 + 16;
    __nv_bfloat16 *a = nullptr, *g = nullptr;
    float *dw = nullptr, *partial = nullptr;
    double *ref = nullptr;
    int *err = nullptr;
    if (cudaMalloc(&a, elems * 2) || cudaMalloc(&g, elems * 2) || cudaMalloc(&dw, 5 * kOut * 4) ||
        cudaMalloc(&partial, (size_t)sms * 28 * 256 * 4) || cudaMalloc(&ref, 256 * 8) || cudaMalloc(&err, 4))
        return 2;
    fill_kernel<<<256, 256>>>(a, ny, rows, 11u);
    fill_kernel<<<256, 256>>>(g, ny, rows, 29u);
    cudaMemset(dw, 0, 5 * kOut * 4);
    cudaMemset(ref, 0, 256 * 8);
    cudaMemset(err, 0, 4);
    const __nv_bfloat16 *as[5] = {a, a, a, a, a}, *gs[5] = {g, g, g, g, g};
    asets::WgradOut out{};
    for (int l = 0; l < 5; ++l) {
        out.dw[l] = dw + l * kOut;
        out.db[l] = out.dw[l] + 27 * 256;
    }
    if (asets::launch_wgrad_layers(reinterpret_cast<asets::EncodeTiledFn>(fn), 5, as, gs, out, ny, nx, nz, partial,
                                   sms, err, 0, 1) != cudaSuccess)
        return 3;
    ref_kernel<<<256, 256>>>(a, g, ny, rows, ref);
    if (cudaDeviceSynchronize() != cudaSuccess)
        return 4;
    int herr = 0;
    cudaMemcpy(&herr, err, 4, cudaMemcpyDeviceToHost);
    std::vector<float> got(5 * kOut);
    std::vector<double> r(256);
    cudaMemcpy(got.data(), dw, got.size() * 4, cudaMemcpyDeviceToHost);
    cudaMemcpy(r.data(), ref, r.size() * 8, cudaMemcpyDeviceToHost);
    double worst = 0.0;
    for (int l = 0; l < 5; ++l)
        for (int i = 0; i < 256; ++i)
            worst = std::fmax(worst, std::fabs(got[l * kOut + 13 * 256 + i] - r[i]) / r[i]);
    *worst_out = worst;
    for (void *p : {(void *)a, (void *)g, (void *)dw, (void *)partial, (void *)ref, (void *)err})
        cudaFree(p);
    return herr ? 5 : 0;
}
