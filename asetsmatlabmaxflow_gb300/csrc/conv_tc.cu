// 3x3x3 convolutions of the learned warm start on the 5th-generation tensor
// cores (tcgen05): BF16 activations and weights, FP32 accumulation in TMEM.
//
// Activations are channels-last, 16 channels of BF16 per voxel
// ([z][x][y][16]).  A convolution is an implicit GEMM: an output tile is 128
// voxels of one z (M = 128), each of the 27 taps is one MMA with K = 16 input
// channels and N = 16 output channels, and the accumulator (128 x 16 FP32)
// lives in TMEM.  One 5D TMA load per tile stages the tile's rows and their
// neighbours, zero-filled outside the volume (the convolution's zero padding),
// as [row][channel half][voxel][8 channels]: the no-swizzle K-major layout in
// which a tap's A operand is a plain offset.
//
// The operand's sixteen groups of eight voxels lie at a fixed distance: a
// tile is eight voxels along y at 16 x, whose neighbourhood is 3 x 18 rows of
// ten voxels (4.2 loaded for each of the tile; 128 along y at one x: 9, and
// three quarters of a tile empty at 32^3).  A layer is bound by its fixed part
// when the volume is small and by the MMAs when it is large (27 at 28 ns a
// tile): 8.3 us at 32^3 and 12 us at 128 x 32 x 32, where a tile of 128 along y
// at one x, loaded in runs of 128 bytes, took 24 and 22.  Two blocks an SM
// overlap one's start and end with the other's work.  Where that fills them
// better, a tile's 16 rows are those of z at one x instead (`along_z`): a call of
// 512 x 1 x 128 39 us against 64.
//
// The same kernel computes the data gradient: with `flip` the taps are
// mirrored and the weight matrix transposed.  The weight gradient is a
// separate tcgen05 kernel (wgrad_tc.cuh).  The epilogue adds the bias and
// an optional FP32 addend (a second convolution's result), then applies ReLU
// and an optional mask (the ReLU derivative of the layer below).
#include <cuda_bf16.h>

#include <cstring>

#include "internal.h"
#include "tcgen05.cuh"

namespace asets {

constexpr int kConvThreads = 192;            // warp 0: TMA, warp 1: MMA, warps 2-5: epilogue
constexpr int kConvStagesLog2 = 2, kConvStages = 1 << kConvStagesLog2;  // deepest TMA ring
constexpr int kConvAcc = 8;                  // TMEM accumulators (16 FP32 columns each)
constexpr int kConvHalfBytes = 10 * 16, kConvRowBytes = 2 * kConvHalfBytes;
constexpr int kConvStageStride = (3 * 18 * kConvRowBytes + 127) / 128 * 128;  // 17,280
constexpr int kConvTapBytes = 2 * 16 * 16;              // B operand of one tap
constexpr int kConvWBytes = 27 * kConvTapBytes;         // 13,824 B
constexpr int kConvSmem = kConvStages * kConvStageStride + kConvWBytes + 128;
static_assert(2 * (kConvSmem + 1024) <= 227 * 1024, "two blocks an SM");

struct ConvTcArgs {
    CUtensorMap act;           // 5D view (8 ch, y, half, x, z) of the BF16 input
    const __nv_bfloat16 *w;    // [27][16 in][16 out]
    const float *bias;         // [16] or null
    const __nv_bfloat16 *mask; // [v][16] or null: output *= (mask > 0)
    const float *addend;       // [v][16] FP32 or null: added before ReLU and mask
    void *out;                 // [v][16] BF16 or FP32
    int *err;
    int ny, nx;                // nx: of the tiles' second axis (x, or z along_z)
    int ytiles, xtiles, ntiles;  // tiles of 8 x 16 voxels
    int step_x, step_r;        // rows of the volume per step of the second axis and of the other
    int tap_z, tap_x;          // bytes per step of a tap's dz and dx in a stage
    int relu, out_fp32, flip;
    int hp_in, hp_out;         // half-planar BF16 input (and mask) / output
    int ypad;                  // half-planar row length (ny rounded up to 8)
    int stages_log2;           // TMA ring depth of this launch
    int stage_bytes;           // of the staged [other axis][second axis][half][voxel][8]
};

// Chained launches (ConvLaunch::chained) start while the layer before still
// runs, as far as its blocks leave room, and do what does not depend on it --
// barriers, tensor memory, the weights' layout -- before they wait for it.
// A block lets its dependents start only once it holds its tensor memory:
// they keep theirs while they wait for this layer, so that a block of it which
// still had to allocate could wait for ever.  A launch takes no more stages than
// its blocks have tiles, so that blocks of both layers fit on an SM.  A training pass at 32^3: 172 -> 143 us, 137 with the
// weight gradients' launch chained too.
//
// Warp-specialised: warp 0 (one lane) keeps a ring of kConvStages tile
// stages loading, warp 1 (one lane) issues each tile's 27 MMAs into one of
// kConvAcc TMEM accumulators as soon as its stage and accumulator are free
// and commits them to the stage's "empty" and the accumulator's "full"
// barrier, and warps 2-5 (TMEM lane quarters 2, 3, 0, 1) drain full
// accumulators through the epilogue and hand them back.  No role waits on
// another's per-tile round trip, so the tensor core sees a steady stream
// of MMAs.  Every wait is bounded; a timeout raises the shared abort flag,
// every role leaves its loop, the producer waits (bounded) for its copies
// in flight and the MMA lane for its last commit before TMEM is freed.
__global__ void __launch_bounds__(kConvThreads, 2) conv3_tc_kernel(const __grid_constant__ ConvTcArgs A)
{
    extern __shared__ __align__(128) unsigned char smem_raw[];
    __shared__ uint64_t full_bar[kConvStages], empty_bar[kConvStages];
    __shared__ uint64_t accf_bar[kConvAcc], acce_bar[kConvAcc];
    __shared__ uint32_t s_tmem;
    __shared__ int s_abort;
    unsigned char *smem = reinterpret_cast<unsigned char *>(
        (reinterpret_cast<uintptr_t>(smem_raw) + 127) & ~static_cast<uintptr_t>(127));
    const int stages = 1 << A.stages_log2, smask = stages - 1;
    unsigned char *wsm = smem + stages * kConvStageStride;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

    if (tid == 0) {
        s_abort = 0;
        for (int i = 0; i < stages; ++i) {
            mbar_init(&full_bar[i], 1);
            mbar_init(&empty_bar[i], 1);
        }
        for (int i = 0; i < kConvAcc; ++i) {
            mbar_init(&accf_bar[i], 1);
            mbar_init(&acce_bar[i], 4);  // one arrival per epilogue warp
        }
        mbar_fence_init();
    }
    if (warp == 1) {
        tmem_alloc(&s_tmem, kConvAcc * 16);
        grid_launch_dependents();  // not before the allocation (above)
    }

    const int ntiles = A.ntiles;
    const int mine = ((int)blockIdx.x < ntiles) ? (ntiles - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;
    auto issue = [&](int j) {
        const int st = j & smask, tile = blockIdx.x + j * gridDim.x;
        const int yt = tile % A.ytiles, rest = tile / A.ytiles;
        const int y = yt * 8, x = rest % A.xtiles * 16, z = rest / A.xtiles;
        mbar_arrive_expect_tx(&full_bar[st], A.stage_bytes);
        tma_load_5d(smem + st * kConvStageStride, &A.act, A.hp_in ? 2 * (y - 1) : 0, A.hp_in ? 0 : y - 1, 0,
                    x - 1, z - 1, &full_bar[st]);
    };
    int issued = 0;
    if (tid == 0) {  // the first tiles load while the other warps lay out the weights
        grid_dependency_wait();
        for (; issued < stages && issued < mine; ++issued)
            issue(issued);
    }

    // B operands: tap t as [k half][n][8 k] (core matrices of 8 n x 8 k).  A
    // thread's eight loads are independent: one round trip each for the five
    // or six groups, where one load per iteration took 36 (a third of a
    // layer's time at 32^3).
#pragma unroll 3
    for (int i = tid - 32; warp > 0 && i < 27 * 32; i += kConvThreads - 32) {
        const int t = i / 32, half = (i / 16) & 1, n = i % 16;
        __align__(16) __nv_bfloat16 v[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            const int k = half * 8 + e;
            v[e] = A.flip ? A.w[(26 - t) * 256 + n * 16 + k] : A.w[t * 256 + k * 16 + n];
        }
        *reinterpret_cast<uint4 *>(wsm + t * kConvTapBytes + half * 256 + n * 16) =
            *reinterpret_cast<const uint4 *>(v);
    }
    fence_proxy_async_smem();
    tc_fence_before_sync();
    grid_dependency_wait();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem = s_tmem;

    if (warp == 0) {
        // ---- producer
        if (lane == 0) {
            for (; issued < mine; ++issued) {
                const int st = issued & smask;
                if (!mbar_wait_bounded(&empty_bar[st], ((issued >> A.stages_log2) - 1) & 1, &s_abort))
                    break;
                issue(issued);
            }
            if (s_abort) {
                // drain the copies in flight of this CTA (bounded)
                volatile int drain_flag = 0;
                for (int j = issued > stages ? issued - stages : 0; j < issued; ++j)
                    mbar_wait_bounded(&full_bar[j & smask], (j >> A.stages_log2) & 1,
                                      (int *)&drain_flag);
            }
        }
    } else if (warp == 1) {
        // ---- MMA issue
        if (lane == 0) {
            const uint32_t idesc = umma_idesc_bf16_f32(128, 16);
            const uint32_t b0 = smem_addr(wsm);
            int done = 0;
            for (int j = 0; j < mine; ++j) {
                const int st = j & smask, slot = j % kConvAcc;
                if (!mbar_wait_bounded(&full_bar[st], (j >> A.stages_log2) & 1, &s_abort))
                    break;
                if (j >= kConvAcc &&
                    !mbar_wait_bounded(&acce_bar[slot], ((j / kConvAcc) - 1) & 1, &s_abort))
                    break;
                tc_fence_after_sync();
                const uint32_t a0 = smem_addr(smem + st * kConvStageStride);
                for (int t = 0; t < 27; ++t) {
                    const int dz = t / 9, dx = (t / 3) % 3, dy = t % 3;
                    const uint32_t a = a0 + dz * A.tap_z + dx * A.tap_x + dy * 16;
                    const uint64_t ad = umma_smem_desc(a, kConvHalfBytes, kConvRowBytes);
                    const uint64_t bd = umma_smem_desc(b0 + t * kConvTapBytes, 256, 128);
                    umma_bf16(tmem + slot * 16, ad, bd, idesc, t > 0 ? 1u : 0u);
                }
                umma_commit(&empty_bar[st]);
                umma_commit(&accf_bar[slot]);
                done = j + 1;
            }
            if (s_abort && done > 0) {
                // the last committed MMAs finish before TMEM is freed (bounded)
                volatile int drain_flag = 0;
                const int j = done - 1;
                mbar_wait_bounded(&accf_bar[j % kConvAcc], (j / kConvAcc) & 1, (int *)&drain_flag);
            }
        }
    } else {
        // ---- epilogue: warp w reads TMEM lanes 32 * (w % 4) .. + 31
        const int q = warp & 3;
        float bias[16];
#pragma unroll
        for (int c = 0; c < 16; ++c)
            bias[c] = A.bias ? __ldg(A.bias + c) : 0.f;
        for (int j = 0; j < mine; ++j) {
            const int slot = j % kConvAcc;
            if (!mbar_wait_bounded(&accf_bar[slot], (j / kConvAcc) & 1, &s_abort))
                break;
            tc_fence_after_sync();
            float acc[16];
            tmem_load16(tmem + ((uint32_t)(32 * q) << 16) + slot * 16, acc);
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0)
                asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr(&acce_bar[slot]))
                             : "memory");
            const int tile = blockIdx.x + j * gridDim.x;
            const int yt = tile % A.ytiles, rest = tile / A.ytiles;
            const int m = 32 * q + lane, z = rest / A.xtiles;
            const int x = rest % A.xtiles * 16 + (m >> 3), y = yt * 8 + (m & 7);
            if (y < A.ny && x < A.nx) {
                const long long zx = (long long)z * A.step_r + (long long)x * A.step_x, v = zx * A.ny + y;
                float o[16];
#pragma unroll
                for (int c = 0; c < 16; ++c)
                    o[c] = acc[c] + bias[c];
                if (A.addend) {
                    const float4 *ap = reinterpret_cast<const float4 *>(A.addend + v * 16);
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        const float4 a4 = __ldg(ap + k);
                        o[4 * k] += a4.x;
                        o[4 * k + 1] += a4.y;
                        o[4 * k + 2] += a4.z;
                        o[4 * k + 3] += a4.w;
                    }
                }
                if (A.relu) {
#pragma unroll
                    for (int c = 0; c < 16; ++c)
                        o[c] = fmaxf(o[c], 0.f);
                }
                // element offsets of the voxel's two channel halves in the input layout
                const long long h0 = A.hp_in ? (zx * 2) * A.ypad * 8 + (long long)y * 8 : v * 16;
                const long long h1 = A.hp_in ? h0 + (long long)A.ypad * 8 : v * 16 + 8;
                if (A.mask) {
                    const uint4 m0 = __ldg(reinterpret_cast<const uint4 *>(A.mask + h0));
                    const uint4 m1 = __ldg(reinterpret_cast<const uint4 *>(A.mask + h1));
                    const __nv_bfloat16 *mb0 = reinterpret_cast<const __nv_bfloat16 *>(&m0);
                    const __nv_bfloat16 *mb1 = reinterpret_cast<const __nv_bfloat16 *>(&m1);
#pragma unroll
                    for (int c = 0; c < 8; ++c) {
                        if (!(__bfloat162float(mb0[c]) > 0.f))
                            o[c] = 0.f;
                        if (!(__bfloat162float(mb1[c]) > 0.f))
                            o[8 + c] = 0.f;
                    }
                }
                if (A.out_fp32) {
                    float4 *op = reinterpret_cast<float4 *>(static_cast<float *>(A.out) + v * 16);
#pragma unroll
                    for (int k = 0; k < 4; ++k)
                        op[k] = make_float4(o[4 * k], o[4 * k + 1], o[4 * k + 2], o[4 * k + 3]);
                } else {
                    __align__(16) __nv_bfloat16 ob[16];
#pragma unroll
                    for (int c = 0; c < 16; ++c)
                        ob[c] = __float2bfloat16_rn(o[c]);
                    __nv_bfloat16 *ob0 = static_cast<__nv_bfloat16 *>(A.out);
                    const long long o0 = A.hp_out ? (zx * 2) * A.ypad * 8 + (long long)y * 8 : v * 16;
                    const long long o1 = A.hp_out ? o0 + (long long)A.ypad * 8 : v * 16 + 8;
                    *reinterpret_cast<uint4 *>(ob0 + o0) = reinterpret_cast<const uint4 *>(ob)[0];
                    *reinterpret_cast<uint4 *>(ob0 + o1) = reinterpret_cast<const uint4 *>(ob)[1];
                }
            }
        }
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    if (tid == 0 && s_abort)
        atomicOr(A.err, 1);
    if (warp == 1)
        tmem_dealloc(tmem, kConvAcc * 16);
}

int conv_smem_bytes() { return kConvSmem; }

cudaError_t launch_conv3_tc(EncodeTiledFn encode, const ConvLaunch &c, int num_sms,
                            cudaStream_t st, int *d_err)
{
    ConvTcArgs A;
    memset(&A, 0, sizeof A);
    // The tiles' second axis (the one of 16 rows) and the other: x and z, or z
    // and x where that makes fewer tiles.
    const bool along_z = (long long)((c.nz + 15) / 16) * c.nx < (long long)((c.nx + 15) / 16) * c.nz;
    const int n2 = along_z ? c.nz : c.nx, n3 = along_z ? c.nx : c.nz;
    // The BF16 input as (8 ch, y, half, second, other) for channels-last
    // [z][x][y][16]; half-planar [z][x][half][ypad][8] as (ypad voxels of two
    // 8-byte elements, 1, half, second, other), so that a box row is one run of
    // memory.  No more rows than a narrow volume has: what stays in the stage
    // from another tile meets only outputs past the volume.
    const int ypad = (c.ny + 7) / 8 * 8, xrows = n2 < 16 ? n2 + 2 : 18;
    const cuuint64_t row = (cuuint64_t)32 * (c.hp_in ? ypad : c.ny);  // bytes of a row of the volume
    const cuuint64_t step2 = along_z ? row * c.nx : row, step3 = along_z ? row : row * c.nx;
    cuuint64_t dims[5], strides[4];
    cuuint32_t box[5];
    if (c.hp_in) {
        const cuuint64_t d[5] = {(cuuint64_t)ypad * 2, 1, 2, (cuuint64_t)n2, (cuuint64_t)n3};
        const cuuint64_t s[4] = {(cuuint64_t)16 * ypad, (cuuint64_t)16 * ypad, step2, step3};
        const cuuint32_t b[5] = {20, 1, 2, (cuuint32_t)xrows, 3};
        memcpy(dims, d, sizeof d);
        memcpy(strides, s, sizeof s);
        memcpy(box, b, sizeof b);
    } else {
        const cuuint64_t d[5] = {8, (cuuint64_t)c.ny, 2, (cuuint64_t)n2, (cuuint64_t)n3};
        const cuuint64_t s[4] = {32, 16, step2, step3};
        const cuuint32_t b[5] = {8, 10, 2, (cuuint32_t)xrows, 3};
        memcpy(dims, d, sizeof d);
        memcpy(strides, s, sizeof s);
        memcpy(box, b, sizeof b);
    }
    cuuint32_t estr[5] = {1, 1, 1, 1, 1};
    CUresult r = encode(&A.act, c.hp_in ? CU_TENSOR_MAP_DATA_TYPE_INT64 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 5,
                        const_cast<void *>(c.x), dims,
                        strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                        CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS)
        return cudaErrorInvalidValue;
    A.w = static_cast<const __nv_bfloat16 *>(c.w);
    A.bias = c.bias;
    A.mask = static_cast<const __nv_bfloat16 *>(c.mask);
    A.addend = c.addend;
    A.out = c.y;
    A.err = d_err;
    A.ny = c.ny;
    A.nx = n2;
    A.ytiles = ypad / 8;
    A.xtiles = (n2 + 15) / 16;
    A.ntiles = A.ytiles * A.xtiles * n3;
    A.step_x = along_z ? c.nx : 1;
    A.step_r = along_z ? 1 : c.nx;
    A.relu = c.relu;
    A.out_fp32 = c.out_fp32;
    A.flip = c.flip;
    A.hp_in = c.hp_in;
    A.hp_out = c.hp_out;
    A.ypad = ypad;
    const int other_bytes = xrows * kConvRowBytes;
    A.tap_z = along_z ? kConvRowBytes : other_bytes;
    A.tap_x = along_z ? other_bytes : kConvRowBytes;
    A.stage_bytes = 3 * other_bytes;
    cudaError_t e = cudaFuncSetAttribute(conv3_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         kConvSmem);
    if (e != cudaSuccess)
        return e;
    const int tiles = A.ntiles, grid = tiles < 2 * num_sms ? tiles : 2 * num_sms;
    while (A.stages_log2 < kConvStagesLog2 && (grid << A.stages_log2) < tiles)
        ++A.stages_log2;
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(kConvThreads);
    cfg.dynamicSmemBytes = (kConvStageStride << A.stages_log2) + kConvWBytes + 128;
    cfg.stream = st;
    cfg.attrs = &attr;
    cfg.numAttrs = c.chained ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, conv3_tc_kernel, A);
}

}  // namespace asets
