// Weight and bias gradients of a 3x3x3, 16 -> 16 channel convolution on the
// 5th-generation tensor cores (tcgen05), BF16 operands, FP32 accumulation.
//
//   dW[t][ci][co] = sum_v a[v + off_t][ci] * g[v][co],   db[co] = sum_v g[v][co]
//
// is, per tap t, a GEMM with the voxels as the reduction axis K:
// D_t[ci][co] = sum_v A_t[v][ci] * G[v][co].  Both operands are read in the
// layout the forward kernel stages (conv_tc.cu): [channel half][voxel][8
// channels], i.e. 8 channels contiguous per voxel -- MN-major operands
// (instruction descriptor bits 15 and 16).  A tap's shift is then an offset
// along the voxels, never along the 16-byte inner dimension the TMA loads
// are aligned on.  The channel halves of the nine staged (dz, dx) rows lie at
// one distance, so the first eight rows of a dy are one MMA's M = 8 rows x 16
// ci; the last row's taps are the M of two more, one a half, whose groups lie
// one voxel apart (three shifts used, the others discarded).  N = 16 co, K =
// 16 voxels.  A sixth MMA with M a constant block of ones gives the bias
// gradient.  6 x 16 FP32 columns of TMEM, five times.  What bounds it is the operands'
// way out of shared memory: 28 MMAs with the gradient as M (16 rows of 128
// used) took 0.78 us per 16 voxels, four of N = 144 0.47, these six 0.18.
//
// Persistent grid, one CTA per SM (the shared memory use keeps it so);
// a CTA walks rows of up to 112 voxels along y, several TMA stages deep; one thread
// issues the row's MMAs (six per 16 voxels, none past the volume's end, where
// the gradient is zero) and the refill of the previous row's stage once
// that row's MMAs have committed.  At the end each CTA writes its 28 x 16 x
// 16 partial sums, and a second kernel adds the CTAs' partials in a fixed
// order into dW and db (deterministic).
#pragma once

#include <cuda_bf16.h>

#include <cstring>

#include "internal.h"
#include "tcgen05.cuh"

namespace asets {

constexpr int kWgtThreads = 128;
constexpr int kWgtMaxStages = 8;
constexpr int kWgtTaps = 28;                               // 27 taps + bias
// An output row is at most 112 voxels, its staged activations y-1 .. y+112
// (114 voxels: what one box row takes, see the tensor maps below).
constexpr int kWgtSpan = 112;
constexpr int kWgtActMax = (9 * 2 * (kWgtSpan + 2) * 16 + 127) / 128 * 128;
constexpr int kWgtGradMax = 2 * kWgtSpan * 16;             // [half][voxel][8 co]
constexpr int kWgtOnesBytes = 16 * 256;                    // [16 M groups][16 voxels][8] ones
// Shared memory: ones, gradient stages, activation stages, and what the last
// row's discarded shifts read past the last one (13 voxels).  Four stages of
// the largest rows; shorter rows leave room for up to eight.
constexpr int kWgtSmem = kWgtOnesBytes + 4 * (kWgtActMax + kWgtGradMax) + 256 + 128;
static_assert(kWgtGradMax % 128 == 0, "stage alignment");
// Accumulators: a CTA's rows go round sets of six, which are added up at the
// end.  With one set, the 30 CTAs a layer of five has would sum five times as
// many voxels in one single-precision chain as 152 CTAs do.
constexpr int kWgtSets = 5, kWgtSetCols = 6 * 16;
constexpr int kWgtTmem = 512;                              // columns: 480 used
static_assert(kWgtSets * kWgtSetCols <= kWgtTmem, "tensor memory of a CTA");
constexpr int kWgtLayers = 5;

struct WgradTcArgs {
    CUtensorMap act[kWgtLayers];   // the BF16 inputs, staged 3x3 rows as [row][half][voxel][8]
    CUtensorMap grad[kWgtLayers];  // the BF16 output gradients, staged [half][voxel][8]
    float *partial;                // [layer][CTA of the layer][28][16 ci][16 co]
    int *err;
    int ny, nx, nz, ytiles;
    int ctas;                      // of a layer
    int hp;                        // half-planar operands
    int act_half, stage_bytes, grad_half, span;
    int stages, act_stride, act_off;         // the shared memory: stages, activations from act_off
};

__global__ void __launch_bounds__(kWgtThreads, 1)
    wgrad_tc_kernel(const __grid_constant__ WgradTcArgs A)
{
    extern __shared__ __align__(128) unsigned char smem_raw[];
    __shared__ uint64_t full_bar[kWgtMaxStages], mma_bar[kWgtMaxStages];
    __shared__ uint32_t s_tmem;
    __shared__ int s_abort;
    unsigned char *smem = reinterpret_cast<unsigned char *>(
        (reinterpret_cast<uintptr_t>(smem_raw) + 127) & ~static_cast<uintptr_t>(127));
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, stages = A.stages;

    if (tid == 0) {
        s_abort = 0;
        for (int i = 0; i < stages; ++i) {
            mbar_init(&full_bar[i], 1);
            mbar_init(&mma_bar[i], 1);
        }
        mbar_fence_init();
    }
    const int ntiles = A.ytiles * A.nx * A.nz;
    // tiles of this CTA: first, first + A.ctas, ... of one layer
    const int layer = blockIdx.x / A.ctas, first = blockIdx.x % A.ctas;
    const int mine = first < ntiles ? (ntiles - 1 - first) / A.ctas + 1 : 0;
    // the producer walks its tiles without a division: a lone thread's chain of
    // them took as long as the tile's MMAs
    int yt = first % A.ytiles, x = first / A.ytiles % A.nx, z = first / A.ytiles / A.nx;
    const int step_y = A.ctas % A.ytiles, step_x = A.ctas / A.ytiles % A.nx, step_z = A.ctas / A.ytiles / A.nx;
    int issued = 0, put = 0;  // tiles issued, the next one's stage
    auto issue = [&]() {
        mbar_arrive_expect_tx(&full_bar[put], A.stage_bytes);
        const int y = yt * A.span;
        tma_load_5d(smem + A.act_off + put * A.act_stride, &A.act[layer], A.hp ? 2 * (y - 1) : 0,
                    A.hp ? 0 : y - 1, 0, x - 1, z - 1, &full_bar[put]);
        tma_load_5d(smem + kWgtOnesBytes + put * kWgtGradMax, &A.grad[layer], A.hp ? 2 * y : 0, A.hp ? 0 : y,
                    0, x, z, &full_bar[put]);
        ++issued;
        put = put + 1 == stages ? 0 : put + 1;
        yt += step_y;
        x += step_x;
        z += step_z;
        if (yt >= A.ytiles) {
            yt -= A.ytiles;
            ++x;
        }
        if (x >= A.nx) {
            x -= A.nx;
            ++z;
        }
    };
    if (tid == 0) {
        grid_dependency_wait();  // a chained launch: as in conv_tc.cu
        while (issued < stages && issued < mine)
            issue();
    }
    // the block of ones (bias gradient), BF16 1.0
    for (int i = tid; i < kWgtOnesBytes / 2; i += kWgtThreads)
        reinterpret_cast<unsigned short *>(smem)[i] = 0x3F80u;
    if (warp == 0)
        tmem_alloc(&s_tmem, kWgtTmem);
    fence_proxy_async_smem();
    tc_fence_before_sync();
    grid_dependency_wait();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem = s_tmem;

    // M = 128, N = 16, both operands MN-major
    const uint32_t idesc = umma_idesc_bf16_f32(128, 16) | (1u << 15) | (1u << 16);

    if (tid == 0) {
        // ---- producer: refills a stage once its MMAs are done
        for (uint32_t ph = 0; issued < mine; ph ^= (put == 0)) {
            if (!mbar_wait_bounded(&mma_bar[put], ph, &s_abort))
                break;
            issue();
        }
        if (s_abort) {
            // drain the copies still in flight (bounded)
            int drain_flag = 0;
            for (int j = issued > stages ? issued - stages : 0; j < issued; ++j)
                mbar_wait_bounded(&full_bar[j % stages], (j / stages) & 1, &drain_flag);
        }
    } else if (tid == 32) {
        // ---- MMA issue
        const uint32_t ones = smem_addr(smem);
        int st = 0, y_left = A.ny - first % A.ytiles * A.span;
        uint32_t ph = 0, d = tmem;  // this row's accumulators
        bool ok = true;
        int j = 0;
        for (; j < mine; ++j) {
            ok = mbar_wait_bounded(&full_bar[st], ph, &s_abort);
            if (!ok)
                break;
            tc_fence_after_sync();
            const uint32_t g0 = smem_addr(smem + kWgtOnesBytes + st * kWgtGradMax);
            const uint32_t a0 = smem_addr(smem + A.act_off + st * A.act_stride);
            const int ksteps = ((y_left < A.span ? y_left : A.span) + 15) / 16;
            for (int ks = 0; ks < ksteps; ++ks) {  // 16 voxels per MMA
                // B: co x voxels, core matrices 8 voxels x 8 co; K step 128 B, N step: half
                const uint64_t bd = umma_smem_desc(g0 + ks * 256, 128, A.grad_half);
                const uint32_t acc = (j >= kWgtSets || ks > 0) ? 1u : 0u;
                const uint32_t a = a0 + ks * 256;
                for (int dy = 0; dy < 3; ++dy)  // M step: a channel half, the rows following one another
                    umma_bf16(d + dy * 16, umma_smem_desc(a + dy * 16, 128, A.act_half), bd, idesc, acc);
                for (int h = 0; h < 2; ++h)     // row 8; M step: a voxel
                    umma_bf16(d + (3 + h) * 16, umma_smem_desc(a + (16 + h) * A.act_half, 128, 16), bd,
                              idesc, acc);
                umma_bf16(d + 5 * 16, umma_smem_desc(ones, 128, 256), bd, idesc, acc);
            }
            umma_commit(&mma_bar[st]);
            d = d == tmem + (kWgtSets - 1) * kWgtSetCols ? tmem : d + kWgtSetCols;
            if (++st == stages) {
                st = 0;
                ph ^= 1;
            }
            y_left -= step_y * A.span;  // the next tile's
            if (y_left <= 0)
                y_left += A.ytiles * A.span;
        }
        // the last row's MMAs (and with them all earlier ones) have finished,
        // also before TMEM is freed after a timeout
        const int last = (st == 0 ? stages : st) - 1;
        int drain_flag = 0;
        if (j > 0)
            mbar_wait_bounded(&mma_bar[last], st == 0 ? ph ^ 1 : ph, ok ? &s_abort : &drain_flag);
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const bool good = !s_abort;
    if (tid == 0 && !good)
        atomicOr(A.err, 1);
    if (good) {
        // TMEM lane m is row m / 16 of the nine, ci = m % 16
        float *P = A.partial + (size_t)blockIdx.x * kWgtTaps * 256;
        const int m = tid;
        auto store = [&](int t, int ci, const float (&v)[16]) {
            float4 *p = reinterpret_cast<float4 *>(P + (t * 16 + ci) * 16);
#pragma unroll
            for (int k = 0; k < 4; ++k)
                p[k] = make_float4(v[4 * k], v[4 * k + 1], v[4 * k + 2], v[4 * k + 3]);
        };
        float v[16];
        const int sets = mine < kWgtSets ? mine : kWgtSets;
        auto load = [&](uint32_t addr) {
            tmem_load16(addr, v);
            for (int i = 1; i < sets; ++i) {
                float w[16];
                tmem_load16(addr + i * kWgtSetCols, w);
#pragma unroll
                for (int k = 0; k < 16; ++k)
                    v[k] += w[k];
            }
        };
        for (int dy = 0; dy < 3; ++dy) {
            load(tmem + ((uint32_t)(32 * warp) << 16) + dy * 16);
            store(m / 16 * 3 + dy, m % 16, v);
        }
        if (warp == 0) {
            for (int h = 0; h < 2; ++h) {  // row 8: lane = 8 * (shift dy) + ci % 8
                load(tmem + (3 + h) * 16);
                if (lane < 24)
                    store(24 + lane / 8, h * 8 + lane % 8, v);
            }
            load(tmem + 5 * 16);
            if (lane == 0)
                store(27, 0, v);  // the bias
        }
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    if (warp == 0)
        tmem_dealloc(tmem, kWgtTmem);
}

// dW[t][ci][co] += sum over a layer's CTAs of the partials (tap 27, ci 0: the
// bias).  Bound by the round trips of a thread's loads: 32 outputs a block,
// and eight threads for each, which add every eighth partial and are then
// added up in order (152 partials: 6 us; one thread for each output: 14).
// blockIdx.y is the layer; its outputs start at dw[layer].
constexpr int kWgtRedOut = 32, kWgtRedSplit = 8;
struct WgradOut {
    float *dw[kWgtLayers], *db[kWgtLayers];
};
__global__ void __launch_bounds__(kWgtRedOut * kWgtRedSplit)
    wgrad_tc_reduce_kernel(const float *partial, int ctas, const WgradOut out)
{
    __shared__ float s_sum[kWgtRedSplit][kWgtRedOut];
    const int o = threadIdx.x % kWgtRedOut, part = threadIdx.x / kWgtRedOut;
    const int i = blockIdx.x * kWgtRedOut + o;  // the bias follows the taps in the partials too
    const float *p = partial + (size_t)blockIdx.y * ctas * kWgtTaps * 256 + i;
    float s = 0.f;
    if (i < 27 * 256 + 16) {
#pragma unroll 8
        for (int b = part; b < ctas; b += kWgtRedSplit)
            s += p[(size_t)b * kWgtTaps * 256];
    }
    s_sum[part][o] = s;
    __syncthreads();
    if (part > 0 || i >= 27 * 256 + 16)
        return;
    for (int q = 1; q < kWgtRedSplit; ++q)
        s += s_sum[q][o];
    if (i < 27 * 256)
        out.dw[blockIdx.y][i] += s;
    else
        out.db[blockIdx.y][i - 27 * 256] += s;
}

// The gradients of `layers` layers of one size, accumulated into out: one
// launch that deals the SMs out to the layers, and one that adds the partial
// sums.  A launch's fixed part is half a layer's time at 32^3, so the five
// layers of the warm-start net take 33 us together against 91 one by one
// (with the former 28 MMAs per 16 voxels: 172).  `partial` holds num_sms x 28 x
// 256 floats.  `hp`: the BF16 arrays half-planar ([z][x][half][y][8]) instead
// of channels-last ([z][x][y][16]).
inline cudaError_t launch_wgrad_layers(EncodeTiledFn encode, int layers, const __nv_bfloat16 *const *act,
                                       const __nv_bfloat16 *const *grad, const WgradOut &out, int ny, int nx,
                                       int nz, float *partial, int num_sms, int *d_err, cudaStream_t st, int hp,
                                       int chained = 0)
{
    if (layers < 1 || layers > kWgtLayers || num_sms < layers)
        return cudaErrorInvalidValue;
    WgradTcArgs A;
    memset(&A, 0, sizeof A);
    const int ypad = (ny + 7) / 8 * 8;
    // rows of equal length, in whole K steps
    const int ytiles = (ny + kWgtSpan - 1) / kWgtSpan, span = ((ny + ytiles - 1) / ytiles + 15) / 16 * 16;
    const int vox = span + 2;  // of an activation row
    // channels-last: (8 ch, y, half, x, z); half-planar [z][x][half][ypad][8]:
    // (ypad voxels of two 8-byte elements, 1, half, x, z), so that a box row
    // is one run of memory.
    cuuint64_t dims[5] = {8, (cuuint64_t)ny, 2, (cuuint64_t)nx, (cuuint64_t)nz};
    cuuint64_t strides[4] = {32, 16, (cuuint64_t)32 * ny, (cuuint64_t)32 * ny * nx};
    cuuint32_t box_a[5] = {8, (cuuint32_t)vox, 2, 3, 3};
    cuuint32_t box_g[5] = {8, (cuuint32_t)span, 2, 1, 1};
    if (hp) {
        const cuuint64_t d[5] = {(cuuint64_t)ypad * 2, 1, 2, (cuuint64_t)nx, (cuuint64_t)nz};
        const cuuint64_t s[4] = {(cuuint64_t)16 * ypad, (cuuint64_t)16 * ypad, (cuuint64_t)32 * ypad,
                                 (cuuint64_t)32 * ypad * nx};
        memcpy(dims, d, sizeof d);
        memcpy(strides, s, sizeof s);
        box_a[0] = 2 * vox;
        box_g[0] = 2 * span;
        box_a[1] = box_g[1] = 1;
    }
    cuuint32_t estr[5] = {1, 1, 1, 1, 1};
    for (int l = 0; l < layers; ++l)
        for (int g = 0; g < 2; ++g)
            if (encode(g ? &A.grad[l] : &A.act[l], hp ? CU_TENSOR_MAP_DATA_TYPE_INT64 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16,
                       5, const_cast<__nv_bfloat16 *>(g ? grad[l] : act[l]), dims, strides, g ? box_g : box_a, estr,
                       CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                       CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                       CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
                return cudaErrorInvalidValue;
    A.partial = partial;
    A.err = d_err;
    A.ny = ny;
    A.nx = nx;
    A.nz = nz;
    A.ytiles = ytiles;
    A.span = span;
    const int tiles = A.ytiles * nx * nz, share = num_sms / layers;
    A.ctas = tiles < share ? tiles : share;
    A.hp = hp;
    A.act_half = vox * 16;
    A.grad_half = span * 16;
    A.stage_bytes = 18 * A.act_half + 2 * A.grad_half;
    A.act_stride = (18 * A.act_half + 127) / 128 * 128;
    A.stages = (kWgtSmem - 128 - kWgtOnesBytes) / (A.act_stride + kWgtGradMax);
    A.stages = A.stages < kWgtMaxStages ? A.stages : kWgtMaxStages;
    A.act_off = kWgtOnesBytes + A.stages * kWgtGradMax;
    cudaError_t e = cudaFuncSetAttribute(wgrad_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kWgtSmem);
    if (e != cudaSuccess)
        return e;
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(A.ctas * layers);
    cfg.blockDim = dim3(kWgtThreads);
    cfg.dynamicSmemBytes = kWgtSmem;
    cfg.stream = st;
    cfg.attrs = &attr;
    cfg.numAttrs = chained ? 1 : 0;
    if ((e = cudaLaunchKernelEx(&cfg, wgrad_tc_kernel, A)) != cudaSuccess)
        return e;
    wgrad_tc_reduce_kernel<<<dim3((27 * 256 + 16 + kWgtRedOut - 1) / kWgtRedOut, layers),
                             kWgtRedOut * kWgtRedSplit, 0, st>>>(partial, A.ctas, out);
    return cudaGetLastError();
}

// One layer.
inline cudaError_t launch_wgrad_tc(EncodeTiledFn encode, const __nv_bfloat16 *act,
                                   const __nv_bfloat16 *grad, float *dw, float *db, int ny, int nx,
                                   int nz, float *partial, int num_sms, int *d_err,
                                   cudaStream_t st, int hp = 0)
{
    WgradOut out{};
    out.dw[0] = dw;
    out.db[0] = db;
    return launch_wgrad_layers(encode, 1, &act, &grad, out, ny, nx, nz, partial, num_sms, d_err, st, hp);
}

}  // namespace asets
