// Matlab-semantics solvers: the GPU form of the reference's Matlab twins of
// the six mex solvers (maxflow/asetsBinaryMF2D.m, asetsBinaryMF3D.m,
// asetsPotts2D.m, asetsPotts3D.m, asetsIshikawa2D.m, asetsIshikawa3D.m),
// the path its tutorials use with gpuArray (tutorials/t03_usingCUDA.m).
// They differ from the mex files: they compute in the class of Ct (single
// or double), break on erriter < beta, initialise Potts/Ishikawa from the
// argmin of Ct, and use Matlab's own expression orders, all kept here;
// the kernels are templated on the element type and follow each .m line's
// evaluation order (IEEE operations, no contraction), so u matches a numpy
// restatement in the same precision bit for bit.
//
// Per iteration, over every flow label (binary 1, Potts L, Ishikawa L-1):
//   1 gradient step of the face flows from ud = divp - ((A - B) + u/cc) of
//     the cell and the one below, (A, B) = (ps, pt) binary, (ps, pt_k)
//     Potts, (pt_k, pt_k+1) Ishikawa; projection factor
//     gk = 1/max(1, |p|/alpha) per cell
//   2 face flows *= 0.5 (gk + gk of the cell below), then per cell divp of
//     every label, the model's sink/source flows and multipliers, erriter and
//     the next iteration's ud; the last block records erriter and the break.
// In double precision u/cc (used by both passes) is kept beside u, divided
// once where u is written.
//
// Bound: single precision by load latency and L2, double by the FP64 pipe.
// Potts 2D 512 x 480 L = 4 in double: 79 us per iteration, 85 with the two launches
// one after another instead of chained; before (four passes, sqrt and division on
// every cell, one thread summing the blocks' errors) 185 us.  Potts 2D 1024^2 L = 4
// in single: 98 us, before 196; binary 512^2 25 (29 not chained).
#include <chrono>
#include <cmath>
#include <cstring>
#include <string>
#include <vector>

#include "asets.h"
#include "device_common.cuh"
#include "div_const.cuh"
#include "internal.h"

using namespace asets;

namespace {

constexpr int kThreads = 256;
enum { MT_BINARY = 0, MT_POTTS = 1, MT_ISHIKAWA = 2 };

struct MTCtl {
    int iter, done, it_num;
    unsigned int ticket;
    int max_it;
    double beta, vol;
};

template <class T>
struct MTArgs {
    int rows, cols, slices, nlab, nflow;
    int step_rows, cell_rows;  // log2 of a tile's rows, where the kernel has no fixed count
    long long n, f1, f2, f3;  // cells and faces per flow label
    T cc, steps, half, one_over_cc, one_over_ccl, beta;
    DivConst<T> by_cc;
    T inv_nlab;           // 1/nlab where nlab is a power of two, else 0
    const T *cs, *ct, *alpha;
    T *u, *ucc, *ud, *pt, *ps, *divp, *gk, *p1, *p2, *p3, *q1, *q2, *q3;
    double *partials;
    T *erriter;
    MTCtl *ctl;
};

template <class T> __device__ __forceinline__ T add(T a, T b);
template <class T> __device__ __forceinline__ T sub(T a, T b);
template <class T> __device__ __forceinline__ T mul(T a, T b);
template <class T> __device__ __forceinline__ T dvd(T a, T b);
template <class T> __device__ __forceinline__ T sqr(T a);
template <> __device__ __forceinline__ float add(float a, float b) { return __fadd_rn(a, b); }
template <> __device__ __forceinline__ float sub(float a, float b) { return __fsub_rn(a, b); }
template <> __device__ __forceinline__ float mul(float a, float b) { return __fmul_rn(a, b); }
template <> __device__ __forceinline__ float dvd(float a, float b) { return __fdiv_rn(a, b); }
template <> __device__ __forceinline__ float sqr(float a) { return __fsqrt_rn(a); }
template <> __device__ __forceinline__ double add(double a, double b) { return __dadd_rn(a, b); }
template <> __device__ __forceinline__ double sub(double a, double b) { return __dsub_rn(a, b); }
template <> __device__ __forceinline__ double mul(double a, double b) { return __dmul_rn(a, b); }
template <> __device__ __forceinline__ double dvd(double a, double b) { return __ddiv_rn(a, b); }
template <> __device__ __forceinline__ double sqr(double a) { return __dsqrt_rn(a); }

// Double precision on this part runs at about 2 operations per clock and SM
// (a warp instruction takes as long as some thirty integer ones), so the
// passes are counted in double operations: what can be decided or formed
// exactly without them is.

// x truncated towards zero to a float, from its bits (magnitude only; below
// 2^-126 gives 0, beyond the float range and for NaN infinity)
__device__ __forceinline__ float mag_f32(double x)
{
    const int hi = __double2hiint(x) & 0x7fffffff;
    const int e = min(max(hi - 0x38000000, 0), 0x0ff00000);
    const unsigned int lo = (e == 0 || e == 0x0ff00000) ? 0u : (unsigned int)__double2loint(x);
    return __uint_as_float(__funnelshift_l(lo, (unsigned int)e, 3));
}
__device__ __forceinline__ bool is_one(double x)
{
    return __double2hiint(x) == 0x3ff00000 && __double2loint(x) == 0;
}

// u/cc of element o: kept beside u in double precision, divided here in single
template <class T>
__device__ __forceinline__ T u_cc(const MTArgs<T> &A, long long o, T u)
{
    if constexpr (sizeof(T) == 8)
        return A.ucc[o];
    else
        return dvd(u, A.cc);
}
template <class T>
__device__ __forceinline__ T u_cc(const MTArgs<T> &A, long long o)
{
    if constexpr (sizeof(T) == 8)
        return A.ucc[o];
    else
        return dvd(A.u[o], A.cc);
}
// stores u of element o (and, in double precision, u/cc beside it);
// returns the new u/cc
template <class T>
__device__ __forceinline__ T set_u(const MTArgs<T> &A, long long o, T v)
{
    A.u[o] = v;
    if constexpr (sizeof(T) == 8) {
        const T q = A.by_cc(v, A.cc);
        A.ucc[o] = q;
        return q;
    } else {
        return dvd(v, A.cc);
    }
}

// Matlab's min(a, b) for ordered values; a NaN a is kept (as the restatement).
// Doubles are compared by their bits as integers (-0 and 0 alike); where an
// exponent is all ones (infinities, NaN) the comparison decides.
__device__ __forceinline__ float mn(float a, float b) { return (a <= b || a != a) ? a : b; }
__device__ __forceinline__ double mn(double a, double b)
{
    const int ha = __double2hiint(a) & 0x7fffffff, hb = __double2hiint(b) & 0x7fffffff;
    if (max(ha, hb) >= 0x7ff00000)
        return (a <= b || a != a) ? a : b;
    const long long ia = __double_as_longlong(a), ib = __double_as_longlong(b);
    const long long low = (long long)0x8000000000000000ull;
    const long long ka = ia < 0 ? low - ia : ia, kb = ib < 0 ? low - ib : ib;
    return ka <= kb ? a : b;
}

// Cell coordinates in 32-bit unsigned arithmetic: every index of a solve
// (cells and faces times labels) is below 2^31 (entry check), and a 64-bit
// division costs several times a 32-bit one.
template <class T>
struct Cell {
    int y, x, z;
    long long g;
    __device__ Cell(const MTArgs<T> &A, long long g_) : g(g_)
    {
        const unsigned int gg = (unsigned int)g_;
        const unsigned int q = gg / (unsigned int)A.rows;
        y = (int)(gg - q * (unsigned int)A.rows);
        const unsigned int z_ = q / (unsigned int)A.cols;
        x = (int)(q - z_ * (unsigned int)A.cols);
        z = (int)z_;
    }
};

// label of the element t of a label-major loop over n cells per label
__device__ __forceinline__ int label_of(long long t, long long n)
{
    return (int)((unsigned int)t / (unsigned int)n);
}
// face arrays: p1 rows x (cols+1) x slices (along columns), p2 (rows+1) x
// cols x slices (along rows), p3 rows x cols x (slices+1) (along slices)
template <class T>
__device__ __forceinline__ long long j1(const MTArgs<T> &A, int y, int x, int z)
{
    return ((long long)z * (A.cols + 1) + x) * A.rows + y;
}
template <class T>
__device__ __forceinline__ long long j2(const MTArgs<T> &A, int y, int x, int z)
{
    return ((long long)z * A.cols + x) * (A.rows + 1) + y;
}
template <class T>
__device__ __forceinline__ long long j3(const MTArgs<T> &A, int y, int x, int z)
{
    return ((long long)z * A.cols + x) * A.rows + y;
}

template <class T>
__device__ __forceinline__ bool finished(const MTArgs<T> &A)
{
    return *(volatile int *)&A.ctl->done != 0;
}

#define MT_LOOP(total)                                                                 \
    for (long long t = blockIdx.x * (long long)kThreads + threadIdx.x; t < (total);    \
         t += (long long)gridDim.x * kThreads)

// ud = divp - ((A - B) + u/cc) of every flow label and cell of the initial
// state, whose flows are zero (and binary ps the same as pt); the cell pass
// forms it for the next iteration
template <class T, int M>
__global__ void mt_ud(const MTArgs<T> A)
{
    MT_LOOP(A.n * A.nflow)
    {
        const long long g = t - (long long)label_of(t, A.n) * A.n;
        const T b = M == MT_ISHIKAWA ? A.pt[t + A.n] : A.pt[t];
        const T a = M == MT_POTTS ? A.ps[g] : A.pt[t];
        A.ud[t] = sub((T)0, add(sub(a, b), u_cc(A, t)));
    }
}

// gradient step of a face flow pp from the ud of the face's upper and lower
// cells: binary pp + steps*(d); Potts/Ishikawa steps*(d) + pp
template <class T, int M>
__device__ __forceinline__ T face_step(const MTArgs<T> &A, T pp, T ud_up, T ud_lo)
{
    const T s = mul(A.steps, sub(ud_up, ud_lo));
    return (M == MT_BINARY) ? add(pp, s) : add(s, pp);
}

// projection rescale of a face flow: 0.5 (gk of the upper cell + gk of the lower) p
template <class T>
__device__ __forceinline__ T face_rescale(const MTArgs<T> &A, T p, T g_up, T g_lo)
{
    return mul(mul(A.half, add(g_up, g_lo)), p);
}

// Whether |p| <= alpha of a cell is sure from a sum of squares in float: the
// magnitudes of its lower and upper faces along columns (a, b), rows (d, e)
// and slices (p, q) are truncated to floats (double; by their bits) or exact
// (single), so with a margin of 2^-18 over all roundings the rounded norm is
// below alpha as well.  Most cells are.
template <class T, int D>
__device__ __forceinline__ bool surely_inside(T a, T b, T d, T e, T p, T q, T al)
{
    auto f = [](T x) {
        if constexpr (sizeof(T) == 8)
            return mag_f32(x);
        else
            return fabsf(x);
    };
    float m = __fmul_rn(f(a), f(a));
    m = __fmaf_rn(f(b), f(b), m);
    m = __fmaf_rn(f(d), f(d), m);
    m = __fmaf_rn(f(e), f(e), m);
    if (D == 3) {
        m = __fmaf_rn(f(p), f(p), m);
        m = __fmaf_rn(f(q), f(q), m);
    }
    const float fa = f(al);
    bool pos;  // above zero and not NaN, which mag_f32 takes for infinity
    if constexpr (sizeof(T) == 8)
        pos = (unsigned long long)__double_as_longlong(al) - 1 < 0x7ff0000000000000ull;
    else
        pos = al > 0.0f;
    return pos && fa > 0x1p-40f && m * (0.5f * (1.0f + 0x1p-18f)) < fa * fa;
}

// projection factor 1/max(1, |p|/alpha) of a cell; 1/1 is exactly 1, so no
// division below alpha
template <class T, int D>
__device__ __forceinline__ T proj_factor(const MTArgs<T> &A, T a, T b, T d, T e, T p, T q, T al)
{
    T s = add(mul(a, a), mul(b, b));
    s = add(s, mul(d, d));
    s = add(s, mul(e, e));
    if (D == 3) {
        s = add(s, mul(p, p));
        s = add(s, mul(q, q));
    }
    const T g = sqr(mul(s, A.half));
    return (g <= al) ? (T)1 : dvd((T)1, dvd(g, al));
}

// ---- the two passes of an iteration --------------------------------------
// The gradient step and the projection factor in one pass, the rescale and
// the cell update in the other.  The stepped flows go to the second face
// buffer (q), the rescaled ones back to p, so that no pass reads a face
// another thread of it writes.

// A block steps the lower faces of a tile of one flow label and slice and
// those of the row and column past it, which the cells' norms share through
// shared memory: a face costs one step (9/8 of one, with the neighbouring tiles'
// faces), which in double is what the pass spends its time on beside the
// norms at capacity.  The upper slice face is stepped again by the cell below it.
//
// Tiles are 32 rows high (ROWS) where that leaves few lanes past the last row; a
// kernel with ROWS = 0 takes 4 to 32 by the launch (tile_rows).
constexpr int kTY = 32, kTX = 8;
static_assert(kTY * kTX == kThreads, "one thread per cell of the tile");
constexpr int kMinRows = 4;

// Rows (a power of two) and columns of a block's tile and its position, tiles
// running along rows, columns, then slices (and labels).
template <class T, int NT, int ROWS>
struct Tile {
    int rows_log2, y0, x0, pl;
    __device__ Tile(const MTArgs<T> &A, int log2) : rows_log2(log2)
    {
        const unsigned int nty = (unsigned int)(A.rows + ty() - 1) / ty();
        const unsigned int ntx = (unsigned int)(A.cols + tx() - 1) / tx();
        const unsigned int q = blockIdx.x / nty;
        y0 = (int)(blockIdx.x % nty) * ty();
        x0 = (int)(q % ntx) * tx();
        pl = (int)(q / ntx);
    }
    __device__ __forceinline__ int ty() const { return ROWS ? ROWS : 1 << rows_log2; }
    __device__ __forceinline__ int tx() const { return ROWS ? NT / (ROWS ? ROWS : 1) : NT >> rows_log2; }
    // row and column of the tile's cell i
    __device__ __forceinline__ int row(int i) const { return i & (ty() - 1); }
    __device__ __forceinline__ int col(int i) const { return ROWS ? i / (ROWS ? ROWS : 1) : i >> rows_log2; }
    static constexpr int kMostTX = NT / (ROWS ? ROWS : kMinRows), kMostTY = ROWS ? ROWS : 32;
};

// Slots in shared memory for the threads of the block that have a rare and
// long piece of work, which full warps then take together: in double a warp
// instruction of the FP64 pipe costs the same for one lane as for all.
// Returns the first slot of the thread's `want` ones (in no fixed order; each
// piece is by itself).
__device__ __forceinline__ int take_slots(int *count, int want)
{
    const int lane = threadIdx.x & 31;
    int before = want;
    for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, before, o);
        if (lane >= o)
            before += v;
    }
    int base = 0;
    if (lane == 31 && before > 0)
        base = atomicAdd(count, before);
    base = __shfl_sync(0xffffffffu, base, 31);
    return base + before - want;
}

template <class T, int M, int D, int ROWS>
__global__ void __launch_bounds__(kThreads) mt_step_gk(const MTArgs<T> A)
{
    constexpr bool QUEUE = sizeof(T) == 8;
    using Q = Tile<T, kThreads, ROWS>;
    // column faces [x][y], row faces [x][y], one past the tile
    __shared__ T s1[kThreads + Q::kMostTY], s2[kThreads + Q::kMostTX];
    __shared__ T s3[QUEUE && D == 3 ? 2 : 1][QUEUE && D == 3 ? kThreads : 1];
    __shared__ unsigned char s_q[kThreads];
    __shared__ int s_n;
    grid_launch_dependents();
    grid_dependency_wait();
    if (finished(A))
        return;
    const Q tile(A, A.step_rows);
    const int ty = tile.ty(), tx = tile.tx(), tid = threadIdx.x;
    const int lane = tile.row(tid), w = tile.col(tid);
    const int k = tile.pl / A.slices, z = tile.pl % A.slices;
    const int y0 = tile.y0, x0 = tile.x0;
    if (threadIdx.x == 0)
        s_n = 0;
    const long long plane = (long long)A.rows * A.cols;
    const T *ud = A.ud + (long long)k * A.n + z * plane;
    const T *f1 = A.p1 + (long long)k * A.f1, *f2 = A.p2 + (long long)k * A.f2;
    // stepped column face (x >= 1) / row face (y >= 1) of cell (y, x); the
    // border faces are zero
    auto step1 = [&](int y, int x) -> T {
        if (y >= A.rows || x < 1 || x >= A.cols)
            return (T)0;
        const T *u = ud + (long long)x * A.rows + y;
        return face_step<T, M>(A, f1[j1(A, y, x, z)], u[0], u[-A.rows]);
    };
    auto step2 = [&](int y, int x) -> T {
        if (x >= A.cols || y < 1 || y >= A.rows)
            return (T)0;
        const T *u = ud + (long long)x * A.rows + y;
        return face_step<T, M>(A, f2[j2(A, y, x, z)], u[0], u[-1]);
    };
    const int y = y0 + lane, x = x0 + w;
    const bool in = y < A.rows && x < A.cols;
    const long long t = (long long)k * A.n + z * plane + (long long)x * A.rows + y;
    const T al = in ? A.alpha[t] : (T)1;
    T p = (T)0, q = (T)0;
    if (D == 3 && in) {
        const T *f3 = A.p3 + (long long)k * A.f3;
        const T v = A.ud[t];
        const T p0 = f3[j3(A, y, x, z)], q0 = f3[j3(A, y, x, z + 1)];
        if (z >= 1) {
            p = face_step<T, M>(A, p0, v, A.ud[t - plane]);
            A.q3[(long long)k * A.f3 + j3(A, y, x, z)] = p;
        }
        if (z + 1 < A.slices)
            q = face_step<T, M>(A, q0, A.ud[t + plane], v);
    }
    const T a = step1(y, x), d = step2(y, x);
    s1[tid] = a;
    s2[tid + w] = d;
    if (tid < ty)
        s1[kThreads + tid] = step1(y, x0 + tx);
    else if (tid - ty < tx)
        s2[(tid - ty) * (ty + 1) + ty] = step2(y0 + ty, x0 + tid - ty);
    if (in && x >= 1)
        A.q1[(long long)k * A.f1 + j1(A, y, x, z)] = a;
    if (in && y >= 1)
        A.q2[(long long)k * A.f2 + j2(A, y, x, z)] = d;
    __syncthreads();
    const T b = s1[tid + ty], e = s2[tid + w + 1];
    const bool inside = !in || surely_inside<T, D>(a, b, d, e, p, q, al);
    if constexpr (QUEUE) {
        if (in && inside)
            A.gk[t] = (T)1;
        const int slot = take_slots(&s_n, inside ? 0 : 1);
        if (!inside) {
            s_q[slot] = (unsigned char)threadIdx.x;
            if (D == 3) {
                s3[0][threadIdx.x] = p;
                s3[D == 3 ? 1 : 0][threadIdx.x] = q;
            }
        }
        __syncthreads();
        if ((int)threadIdx.x < s_n) {  // at most one each
            const int c = s_q[threadIdx.x], cl = tile.row(c), cw = tile.col(c);
            const long long tc = t + (long long)(cw - w) * A.rows + (cl - lane);
            const T pz = D == 3 ? s3[0][c] : (T)0, qz = D == 3 ? s3[D == 3 ? 1 : 0][c] : (T)0;
            A.gk[tc] = proj_factor<T, D>(A, s1[c], s1[c + ty], s2[c + cw], s2[c + cw + 1], pz, qz, A.alpha[tc]);
        }
    } else if (in) {
        A.gk[t] = inside ? (T)1 : proj_factor<T, D>(A, a, b, d, e, p, q, al);
    }
}

// A cell's value of a per-cell array with those of its lower and upper
// neighbours along each axis, and the cell's lower and upper faces of the
// three face arrays, all loaded before any is used (the pass is bound by
// the latency of these loads).  A neighbour outside the volume reads the
// cell itself; its value is not used.
template <class T, int D>
struct Around {
    T v, xl, xu, yl, yu, zl, zu;  // per-cell values
    T a, b, d, e, p, q;           // faces: x lower/upper, y lower/upper, z lower/upper
    long long fa, fd, fp;         // the lower faces' indices
    bool has_xl, has_xu, has_yl, has_yu, has_zl, has_zu;
    __device__ __forceinline__ Around(const MTArgs<T> &A, const Cell<T> &c, const T *cell,
                                      const T *f1, const T *f2, const T *f3)
    {
        const long long g = c.g, pl = (long long)A.rows * A.cols;
        has_xl = c.x >= 1;
        has_xu = c.x + 1 < A.cols;
        has_yl = c.y >= 1;
        has_yu = c.y + 1 < A.rows;
        has_zl = D == 3 && c.z >= 1;
        has_zu = D == 3 && c.z + 1 < A.slices;
        fa = j1(A, c.y, c.x, c.z);
        fd = j2(A, c.y, c.x, c.z);
        fp = j3(A, c.y, c.x, c.z);
        v = cell[g];
        xl = cell[has_xl ? g - A.rows : g];
        xu = cell[has_xu ? g + A.rows : g];
        yl = cell[has_yl ? g - 1 : g];
        yu = cell[has_yu ? g + 1 : g];
        a = f1[fa];
        b = f1[j1(A, c.y, c.x + 1, c.z)];
        d = f2[fd];
        e = f2[j2(A, c.y + 1, c.x, c.z)];
        if (D == 3) {
            zl = cell[has_zl ? g - pl : g];
            zu = cell[has_zu ? g + pl : g];
            p = f3[fp];
            q = f3[j3(A, c.y, c.x, c.z + 1)];
        } else {
            zl = zu = p = q = (T)0;  // no slices: unused
        }
    }
};

// divergence of flow label k at cell c from the stepped flows (q), with the
// rescale of every face; the cell's lower faces are stored (into p)
template <class T, int D>
__device__ __forceinline__ T rescaled_divergence(const MTArgs<T> &A, int k, const Cell<T> &c)
{
    const Around<T, D> s(A, c, A.gk + (long long)k * A.n, A.q1 + (long long)k * A.f1,
                         A.q2 + (long long)k * A.f2, A.q3 + (long long)k * A.f3);
    T a = s.a, b = s.b, d = s.d, e = s.e;
    if (s.has_xl) {
        a = face_rescale(A, a, s.v, s.xl);
        A.p1[(long long)k * A.f1 + s.fa] = a;
    }
    if (s.has_xu)
        b = face_rescale(A, b, s.xu, s.v);
    if (s.has_yl) {
        d = face_rescale(A, d, s.v, s.yl);
        A.p2[(long long)k * A.f2 + s.fd] = d;
    }
    if (s.has_yu)
        e = face_rescale(A, e, s.yu, s.v);
    T dv = sub(b, a);
    dv = add(dv, e);
    dv = sub(dv, d);
    if (D == 3) {
        T p = s.p, q = s.q;
        if (s.has_zl) {
            p = face_rescale(A, p, s.v, s.zl);
            A.p3[(long long)k * A.f3 + s.fp] = p;
        }
        if (s.has_zu)
            q = face_rescale(A, q, s.zu, s.v);
        dv = add(dv, q);
        dv = sub(dv, p);
    }
    return dv;
}

// The same for every cell of a block's tile (double): each face of the tile
// and of the row and column past it is rescaled once, into shared memory, and
// the faces with a factor below 1 by full warps together.  Called by every
// thread of the block.
template <class T, int D, int NT, int ROWS>
struct FaceTile {
    using Q = Tile<T, NT, ROWS>;
    static_assert(NT % 32 == 0 && Q::kMostTX + Q::kMostTY <= NT, "a thread has one face past the tile at most");
    // column faces [x][y], row faces [x][y], one past the tile, slice faces (lower, upper)
    static constexpr int kRow = NT + Q::kMostTY, kSlice = kRow + NT + Q::kMostTX;
    static constexpr int kFaces = kSlice + (D == 3 ? 2 * NT : 0);
    T f[kFaces];
    T g[kFaces][2];            // factors of the faces in the queue
    unsigned short q[kFaces];  // their places in f
    int n;

    // `in`: the thread's cell (y, x, z) is in the volume
    __device__ T divergence(const MTArgs<T> &A, const Q &tile, int k, int y, int x, int z, bool in)
    {
        const int ty = tile.ty(), tx = tile.tx(), tid = threadIdx.x;
        const long long plane = (long long)A.rows * A.cols;
        const T *gk = A.gk + (long long)k * A.n + z * plane;
        const T *q1 = A.q1 + (long long)k * A.f1, *q2 = A.q2 + (long long)k * A.f2;
        const int my1 = tid, my2 = kRow + tid + tile.col(tid);
        // up to five faces a thread: (place, factors), not yet in the queue
        int want = 0, at[5];
        T gu[5], gl[5];
        auto put = [&](int i, int place, bool on, T p, T g_up, T g_lo) {
            f[place] = on ? p : (T)0;
            at[i] = (on && !(is_one(g_up) && is_one(g_lo))) ? place : -1;
            gu[i] = g_up;
            gl[i] = g_lo;
            want += at[i] >= 0;
        };
        auto col = [&](int i, int place, int yy, int xx) {
            const bool on = yy < A.rows && xx >= 1 && xx < A.cols;
            const T *g0 = gk + (long long)xx * A.rows + yy;
            put(i, place, on, on ? q1[j1(A, yy, xx, z)] : (T)0, on ? g0[0] : (T)1,
                on ? g0[-A.rows] : (T)1);
        };
        auto row = [&](int i, int place, int yy, int xx) {
            const bool on = xx < A.cols && yy >= 1 && yy < A.rows;
            const T *g0 = gk + (long long)xx * A.rows + yy;
            put(i, place, on, on ? q2[j2(A, yy, xx, z)] : (T)0, on ? g0[0] : (T)1, on ? g0[-1] : (T)1);
        };
        if (threadIdx.x == 0)
            n = 0;
        __syncthreads();  // and the previous label's faces are read
        col(0, my1, y, x);
        row(1, my2, y, x);
        at[2] = at[3] = at[4] = -1;
        if (tid < ty)
            col(2, NT + tid, y, x + tx);
        else if (tid - ty < tx)
            row(2, kRow + (tid - ty) * (ty + 1) + ty, tile.y0 + ty, tile.x0 + tid - ty);
        if (D == 3) {
            const T *q3 = A.q3 + (long long)k * A.f3;
            const T *g0 = gk + (long long)x * A.rows + y;
            const bool lo = in && z >= 1, up = in && z + 1 < A.slices;
            const T gc = in ? g0[0] : (T)1;
            put(3, kSlice + (int)threadIdx.x, lo, lo ? q3[j3(A, y, x, z)] : (T)0, gc,
                lo ? g0[-plane] : (T)1);
            put(4, kSlice + NT + (int)threadIdx.x, up, up ? q3[j3(A, y, x, z + 1)] : (T)0,
                up ? g0[plane] : (T)1, gc);
        }
        int slot = take_slots(&n, want);
#pragma unroll
        for (int i = 0; i < 5; ++i)
            if (at[i] >= 0) {
                q[slot] = (unsigned short)at[i];
                g[slot][0] = gu[i];
                g[slot][1] = gl[i];
                ++slot;
            }
        __syncthreads();
        const int m = n;
        for (int i = threadIdx.x; i < m; i += NT)
            f[q[i]] = mul(mul(A.half, add(g[i][0], g[i][1])), f[q[i]]);
        __syncthreads();
        const T a = f[my1], b = f[my1 + ty], d = f[my2], e = f[my2 + 1];
        if (in && x >= 1)
            A.p1[(long long)k * A.f1 + j1(A, y, x, z)] = a;
        if (in && y >= 1)
            A.p2[(long long)k * A.f2 + j2(A, y, x, z)] = d;
        T dv = sub(b, a);
        dv = add(dv, e);
        dv = sub(dv, d);
        if (D == 3) {
            const T p = f[kSlice + threadIdx.x], pu = f[kSlice + NT + threadIdx.x];
            if (in && z >= 1)
                A.p3[(long long)k * A.f3 + j3(A, y, x, z)] = p;
            dv = add(dv, pu);
            dv = sub(dv, p);
        }
        return dv;
    }
};

// ---- the cell update --------------------------------------------------------

// binary: ps, pt, u of cell g from its divp dv and old u, pt, Cs, Ct, then
// the next iteration's ud; returns |erru|
template <class T>
__device__ __forceinline__ double binary_update(const MTArgs<T> &A, long long g, T dv, T u, T uc,
                                                T pt0, T cs, T ct)
{
    const T ps = mn(add(sub(add(dv, pt0), uc), A.one_over_cc), cs);
    const T pt = mn(add(add(-dv, ps), uc), ct);
    const T e = mul(A.cc, sub(add(dv, pt), ps));
    A.pt[g] = pt;
    const T q = set_u(A, g, sub(u, e));
    A.ud[g] = sub(dv, add(sub(ps, pt), q));
    return fabs((double)e);
}

// Potts with LFIX labels (0: any): divp and the sink flow of every label,
// the source flow, then the multipliers and the next iteration's ud.  With
// LFIX the labels' values stay in registers and their loads are in flight
// together.
template <class T, int LFIX, class Div>
__device__ __forceinline__ double potts_update(const MTArgs<T> &A, long long g, bool in, Div div)
{
    const long long n = A.n;
    const int L = LFIX > 0 ? LFIX : A.nlab;
    constexpr int R = LFIX > 0 ? LFIX : 1;
    const T ps = in ? A.ps[g] : (T)0;
    T dd[R], pp[R], uu[R];
    T pd = (T)0;
    double err = 0.0;
#pragma unroll
    for (int k = 0; k < L; ++k) {
        const long long o = (long long)k * n + g;
        const T u = in ? A.u[o] : (T)0, uc = in ? u_cc(A, o, u) : (T)0, ct = in ? A.ct[o] : (T)0;
        const T dv = div(k);
        const T pt = mn(add(add(-dv, ps), uc), ct);
        if constexpr (LFIX > 0) {
            dd[k] = dv;
            pp[k] = pt;
            uu[k] = u;
        } else if (in) {
            A.divp[o] = dv;
            A.pt[o] = pt;
        }
        pd = add(pd, sub(add(dv, pt), uc));
    }
    if (!in)
        return 0.0;
    // times 1/nlab where that is exact (a power of two)
    const T mean = A.inv_nlab != (T)0 ? mul(pd, A.inv_nlab) : dvd(pd, (T)A.nlab);
    const T psn = add(mean, A.one_over_ccl);
    A.ps[g] = psn;
#pragma unroll
    for (int k = 0; k < L; ++k) {
        const long long o = (long long)k * n + g;
        const T dv = LFIX > 0 ? dd[LFIX > 0 ? k : 0] : A.divp[o];
        const T pt = LFIX > 0 ? pp[LFIX > 0 ? k : 0] : A.pt[o];
        const T u = LFIX > 0 ? uu[LFIX > 0 ? k : 0] : A.u[o];
        const T e = mul(A.cc, sub(add(dv, pt), psn));
        const T q = set_u(A, o, sub(u, e));
        A.ud[o] = sub(dv, add(sub(psn, pt), q));
        err += fabs((double)e);
    }
    return err;
}

// Ishikawa: divp of every layer, the sink-flow chain (lowest first, each
// layer with the new one below), the multipliers and the next ud of the layer
// below as soon as both of its sink flows are there.
template <class T, class Div>
__device__ __forceinline__ double ishikawa_update(const MTArgs<T> &A, long long g, bool in, Div div)
{
    const long long n = A.n;
    const int L = A.nlab;
    double err = 0.0;
    T dv_b = (T)0, pt_b = (T)0, uc_b = (T)0, u_b = (T)0;  // layer k-1
    for (int k = 0; k < L; ++k) {
        const long long o = (long long)k * n + g;
        T dv = (T)0, u = (T)0, uc = (T)0, up = (T)0, v;
        const T ct = in ? A.ct[o] : (T)0;
        if (k < L - 1) {
            if (in) {
                u = A.u[o];
                uc = u_cc(A, o, u);
                up = A.pt[o + n];
            }
            dv = div(k);
        }
        if (!in)
            continue;
        if (k == 0) {
            v = add(sub(add(dv, up), uc), A.one_over_cc);
        } else {
            v = add(add(-dv_b, pt_b), uc_b);
            if (k < L - 1)
                v = mul(sub(add(add(v, dv), up), uc), (T)0.5);  // v/2 exactly
        }
        const T pt = mn(v, ct);
        A.pt[o] = pt;
        if (k > 0) {
            const T e = mul(A.cc, sub(add(dv_b, pt), pt_b));
            const T q = set_u(A, o - n, sub(u_b, e));
            A.ud[o - n] = sub(dv_b, add(sub(pt_b, pt), q));
            err += fabs((double)e);
        }
        dv_b = dv;
        pt_b = pt;
        uc_b = uc;
        u_b = u;
    }
    return err;
}

// Per cell: divp of every flow label with the rescale of the stepped flows,
// the cell update; the last block records erriter and the break.  Single
// precision strides over the cells; in double a block has a tile (FaceTile).
template <class T, int M, int D, int LFIX, int NT, int ROWS>
__global__ void __launch_bounds__(NT, 1024 / NT) mt_cell(const MTArgs<T> A)
{
    __shared__ double s_red[NT / 32];
    __shared__ int s_last;
    grid_launch_dependents();
    grid_dependency_wait();
    if (finished(A))
        return;
    const int it = *(volatile int *)&A.ctl->iter;
    double err = 0.0;
    auto update = [&](long long t, bool in, auto div) {
        if constexpr (M == MT_BINARY) {
            // the cell's own operands are loaded with the divergence's
            const T u = in ? A.u[t] : (T)0, uc = in ? u_cc(A, t, u) : (T)0, pt = in ? A.pt[t] : (T)0;
            const T cs = in ? A.cs[t] : (T)0, ct = in ? A.ct[t] : (T)0;
            const T dv = div(0);
            if (in)
                err += binary_update(A, t, dv, u, uc, pt, cs, ct);
        } else if constexpr (M == MT_POTTS) {
            err += potts_update<T, LFIX>(A, t, in, div);
        } else {
            err += ishikawa_update<T>(A, t, in, div);
        }
    };
    if constexpr (sizeof(T) == 8) {
        __shared__ FaceTile<T, D, NT, ROWS> faces;
        const Tile<T, NT, ROWS> tile(A, A.cell_rows);
        const int y = tile.y0 + tile.row(threadIdx.x), x = tile.x0 + tile.col(threadIdx.x), z = tile.pl;
        const bool in = y < A.rows && x < A.cols;
        update(((long long)z * A.cols + x) * A.rows + y, in,
               [&](int k) { return faces.divergence(A, tile, k, y, x, z, in); });
    } else {
        MT_LOOP(A.n)
        {
            const Cell<T> c(A, t);
            update(t, true, [&](int k) { return rescaled_divergence<T, D>(A, k, c); });
        }
    }
    for (int o = 16; o > 0; o >>= 1)
        err += __shfl_xor_sync(0xffffffffu, err, o);
    if ((threadIdx.x & 31) == 0)
        s_red[threadIdx.x >> 5] = err;
    __syncthreads();
    if (threadIdx.x == 0) {
        double b = 0.0;
        for (int w = 0; w < NT / 32; ++w)
            b += s_red[w];
        A.partials[blockIdx.x] = b;
        __threadfence();
        s_last = (atomicAdd(&A.ctl->ticket, 1u) == gridDim.x - 1);
    }
    __syncthreads();
    if (!s_last)
        return;
    // the blocks' sums in a fixed order, by every thread of the last block
    // (one thread alone would take longer than the pass at 10^6 cells)
    __threadfence();
    double tot = 0.0;
    for (unsigned int b = threadIdx.x; b < gridDim.x; b += NT)
        tot += __ldcg(A.partials + b);
    for (int o = 16; o > 0; o >>= 1)
        tot += __shfl_xor_sync(0xffffffffu, tot, o);
    __syncthreads();  // s_red is read above by thread 0
    if ((threadIdx.x & 31) == 0)
        s_red[threadIdx.x >> 5] = tot;
    __syncthreads();
    if (threadIdx.x == 0) {
        tot = 0.0;
        for (int w = 0; w < NT / 32; ++w)
            tot += s_red[w];
        const T e = (T)(tot / A.ctl->vol);
        A.erriter[it] = e;
        if (e < A.beta) {
            A.ctl->done = 1;
            A.ctl->it_num = it + 1;
        } else if (it + 1 >= A.ctl->max_it) {
            A.ctl->done = 1;
            A.ctl->it_num = A.ctl->max_it;
        }
        A.ctl->ticket = 0;
        A.ctl->iter = it + 1;
        __threadfence();
    }
}

// initial state (the .m files before their loop)
template <class T, int M>
__global__ void mt_init(const MTArgs<T> A)
{
    MT_LOOP(A.n)
    {
        const long long g = t, n = A.n;
        if (M == MT_BINARY) {
            const T cs = A.cs[g], ct = A.ct[g];
            set_u(A, g, (sub(cs, ct) >= (T)0) ? (T)1 : (T)0);
            A.pt[g] = mn(cs, ct);
            continue;
        }
        // [m, I] = min(Ct, [], labels): the first minimum
        T m = A.ct[g];
        int I = 0;
        for (int k = 1; k < A.nlab; ++k) {
            const T v = A.ct[(long long)k * n + g];
            if (v < m) {
                m = v;
                I = k;
            }
        }
        for (int k = 0; k < A.nlab; ++k)
            A.pt[(long long)k * n + g] = m;
        if (M == MT_POTTS) {
            A.ps[g] = m;
            for (int k = 0; k < A.nlab; ++k)
                set_u(A, (long long)k * n + g, (I == k) ? (T)1 : (T)0);
        } else {
            for (int k = 0; k < A.nlab - 1; ++k)  // u(:,:,k) = init > k, 1-based
                set_u(A, (long long)k * n + g, (I > k) ? (T)1 : (T)0);
        }
    }
}

int mt_grid(long long n, int sms)
{
    long long b = (n + kThreads - 1) / kThreads;
    const long long cap = (long long)sms * 8;
    return (int)(b < 1 ? 1 : (b < cap ? b : cap));
}

// Label counts with a Potts update of their own, which needs no divp
constexpr bool potts_kernel_labels(int nlab) { return nlab >= 2 && nlab <= 6; }

template <class T, int M, int D, int NT, int ROWS>
void launch_cell(const MTArgs<T> &A, int grid, cudaStream_t st)
{
    auto launch = [&](auto kernel) { launch_chained(kernel, dim3(grid), NT, 0, st, A); };
    if constexpr (M == MT_POTTS) {
        switch (A.nlab) {
        case 2: launch(mt_cell<T, M, D, 2, NT, ROWS>); return;
        case 3: launch(mt_cell<T, M, D, 3, NT, ROWS>); return;
        case 4: launch(mt_cell<T, M, D, 4, NT, ROWS>); return;
        case 5: launch(mt_cell<T, M, D, 5, NT, ROWS>); return;
        case 6: launch(mt_cell<T, M, D, 6, NT, ROWS>); return;
        default: break;
        }
    }
    launch(mt_cell<T, M, D, 0, NT, ROWS>);
}

template <class T, int M, int D>
asets_status mt_run(asets_context *ctx, int rows, int cols, int slices, int nlab,
                    const void *Cs, const void *Ct, const void *alpha, int iterNum, double beta,
                    double cc, double steps, void *u_out, void *err_out, int *itNum)
{
    cudaStream_t st = context_stream(ctx);
    const int sms = context_num_sms(ctx);
    MTArgs<T> A;
    memset(&A, 0, sizeof A);
    A.rows = rows;
    A.cols = cols;
    A.slices = slices;
    A.nlab = (M == MT_BINARY) ? 1 : nlab;
    A.nflow = (M == MT_ISHIKAWA) ? nlab - 1 : A.nlab;
    const long long n = (long long)rows * cols * slices;
    A.n = n;
    A.f1 = (long long)rows * (cols + 1) * slices;
    A.f2 = (long long)(rows + 1) * cols * slices;
    A.f3 = D == 3 ? (long long)rows * cols * (slices + 1) : 0;
    // scalars rounded to the class of Ct, as Matlab combines them
    A.cc = (T)cc;
    A.steps = (T)steps;
    A.half = (T)0.5;
    A.one_over_cc = (T)(1.0 / cc);
    A.one_over_ccl = (T)(1.0 / (cc * A.nlab));
    A.beta = (T)beta;
    A.by_cc.set(A.cc);
    A.inv_nlab = (A.nlab & (A.nlab - 1)) == 0 ? (T)1 / (T)A.nlab : (T)0;
    const int nct = A.nlab, nu = (M == MT_ISHIKAWA) ? nlab - 1 : A.nlab;
    const int npt = A.nlab;
    std::vector<void *> bufs;
    auto get = [&](T **p, long long count) {
        void *v = nullptr;
        if (cudaMallocAsync(&v, (size_t)(count < 1 ? 1 : count) * sizeof(T), st) != cudaSuccess)
            return false;
        bufs.push_back(v);
        *p = static_cast<T *>(v);
        return true;
    };
    T *cs = nullptr, *ct = nullptr, *al = nullptr;
    asets_status status = ASETS_OK;
    const int grid = mt_grid(n * A.nflow, sms);
    // Tiles of a slice's cells, and the rows of a tile of nt threads (as log2)
    // that leaves the fewest lanes past the last row and column.
    const auto tiles_of = [&](int ty, int tx) {
        return (long long)((rows + ty - 1) / ty) * ((cols + tx - 1) / tx) * slices;
    };
    const auto best_rows = [&](int nt) {
        int best = 5;
        for (int l = 4; 1 << l >= kMinRows; --l)
            if (tiles_of(1 << l, nt >> l) < tiles_of(1 << best, nt >> best))
                best = l;
        return best;
    };
    // A fixed 32 rows unless others save a seventh of the lanes.
    const long long tiles = tiles_of(kTY, kTX);
    A.step_rows = best_rows(kThreads);
    const long long fitted = tiles_of(1 << A.step_rows, kThreads >> A.step_rows);
    const bool fit_step = 7 * fitted <= 6 * tiles;
    const long long step_tiles = fit_step ? fitted : tiles;
    // The cell update's tiles in double, 32 x 8; a tile's time is its chain of
    // labels and its FP64 operations on one SM, so that small volumes take half
    // ones: with less than a tile an SM 32 x 4 (us an iteration, 8 | 4 columns: 27 x
    // 28 x 21 Potts L = 3, 84 tiles, 41.6 | 31.1; 181 x 64 L = 5, 48 tiles, 31.1 |
    // 27.9), with less than four 16 x 8 where these leave a fifth fewer lanes
    // past the last row (35 x 30 x 19 L = 3: 47.8 | 38.8).
    const int rows32 = (rows + 31) / 32 * 32, rows16 = (rows + 15) / 16 * 16;
    const bool short_tiles = sizeof(T) == 8 && tiles < 4 * sms && 5 * rows16 <= 4 * rows32;
    const bool half_tiles = sizeof(T) == 8 && tiles < sms && !short_tiles;
    const long long cell_tiles = short_tiles ? tiles_of(16, kTX) : half_tiles ? tiles_of(kTY, kTX / 2) : tiles;
    A.cell_rows = best_rows(kThreads / 2);
    const long long fitted_cells = tiles_of(1 << A.cell_rows, (kThreads / 2) >> A.cell_rows);
    const bool fit_cell =
        sizeof(T) == 8 && 7 * fitted_cells <= 6 * cell_tiles * (short_tiles || half_tiles ? 1 : 2);
    const int gcell = sizeof(T) == 8 ? (int)(fit_cell ? fitted_cells : cell_tiles) : mt_grid(n, sms),
              ginit = mt_grid(n, sms);
    bool ok = get(&ct, n * nct) && get(&al, n * A.nflow) && get(&A.u, n * nu) &&
              get(&A.ud, n * A.nflow) &&
              get(&A.q1, A.f1 * A.nflow) && get(&A.q2, A.f2 * A.nflow) && get(&A.q3, A.f3 * A.nflow) &&
              (sizeof(T) != 8 || get(&A.ucc, n * nu)) && get(&A.pt, n * npt) &&
              (M != MT_POTTS || (get(&A.ps, n) && (potts_kernel_labels(nlab) || get(&A.divp, n * nlab)))) &&
              get(&A.gk, n * A.nflow) && get(&A.p1, A.f1 * A.nflow) && get(&A.p2, A.f2 * A.nflow) &&
              get(&A.p3, A.f3 * A.nflow) && get(&A.erriter, iterNum) &&
              (M != MT_BINARY || get(&cs, n));
    void *pv = nullptr;
    ok = ok && cudaMallocAsync(&pv, sizeof(MTCtl) + (size_t)gcell * sizeof(double), st) == cudaSuccess;
    if (ok) {
        bufs.push_back(pv);
        A.ctl = static_cast<MTCtl *>(pv);
        A.partials = reinterpret_cast<double *>(static_cast<char *>(pv) + sizeof(MTCtl));
    }
    cudaError_t e = cudaSuccess;
    MTCtl c0;
    memset(&c0, 0, sizeof c0);
    c0.max_it = iterNum;
    c0.beta = beta;
    c0.vol = (M == MT_BINARY)    ? (double)n
             : (M == MT_POTTS)   ? (double)(n * nlab)
                                 : (double)(n * nlab - 1);  // rows*cols*nlab-1, as the .m files
    if (!ok) {
        status = ASETS_ERR_OUT_OF_MEMORY;
        set_last_error("Matlab-semantics solver: out of device memory");
    } else {
        e = cudaMemcpyAsync(ct, Ct, sizeof(T) * n * nct, cudaMemcpyHostToDevice, st);
        if (e == cudaSuccess)
            e = cudaMemcpyAsync(al, alpha, sizeof(T) * n * A.nflow, cudaMemcpyHostToDevice, st);
        if (e == cudaSuccess && M == MT_BINARY)
            e = cudaMemcpyAsync(cs, Cs, sizeof(T) * n, cudaMemcpyHostToDevice, st);
        if (e == cudaSuccess)
            e = cudaMemcpyAsync(A.ctl, &c0, sizeof c0, cudaMemcpyHostToDevice, st);
        // the flows and the second face buffer start at zero; their border
        // faces are never written and stay zero (the zero-flux border)
        T *zero[] = {A.p1, A.p2, A.p3, A.erriter, A.q1, A.q2, A.q3};
        const long long fn = A.nflow;
        const long long zn[] = {A.f1 * fn, A.f2 * fn, A.f3 * fn, (long long)iterNum, A.f1 * fn, A.f2 * fn, A.f3 * fn};
        for (int i = 0; i < 7 && e == cudaSuccess; ++i)
            if (zn[i] > 0)
                e = cudaMemsetAsync(zero[i], 0, sizeof(T) * zn[i], st);
        A.cs = cs;
        A.ct = ct;
        A.alpha = al;
        if (e == cudaSuccess) {
            mt_init<T, M><<<ginit, kThreads, 0, st>>>(A);
            mt_ud<T, M><<<grid, kThreads, 0, st>>>(A);
            e = cudaGetLastError();
        }
        constexpr int kChunk = 16;
        int h_done = 0;
        for (int done_it = 0; e == cudaSuccess && done_it < iterNum; done_it += kChunk) {
            for (int i = 0; i < kChunk && done_it + i < iterNum; ++i) {
                const dim3 gstep((unsigned int)(step_tiles * A.nflow));
                if (fit_step)
                    launch_chained(mt_step_gk<T, M, D, 0>, gstep, kThreads, 0, st, A);
                else
                    launch_chained(mt_step_gk<T, M, D, kTY>, gstep, kThreads, 0, st, A);
                if constexpr (sizeof(T) == 8) {
                    if (fit_cell)
                        launch_cell<T, M, D, kThreads / 2, 0>(A, gcell, st);
                    else if (short_tiles)
                        launch_cell<T, M, D, kThreads / 2, 16>(A, gcell, st);
                    else if (half_tiles)
                        launch_cell<T, M, D, kThreads / 2, kTY>(A, gcell, st);
                    else
                        launch_cell<T, M, D, kThreads, kTY>(A, gcell, st);
                } else {
                    launch_cell<T, M, D, kThreads, kTY>(A, gcell, st);
                }
            }
            e = cudaGetLastError();
            if (e == cudaSuccess)
                e = cudaMemcpyAsync(&h_done, &A.ctl->done, sizeof(int), cudaMemcpyDeviceToHost, st);
            if (e == cudaSuccess)
                e = cudaStreamSynchronize(st);
            if (h_done)
                break;
        }
        MTCtl out;
        memset(&out, 0, sizeof out);
        if (e == cudaSuccess)
            e = cudaMemcpyAsync(&out, A.ctl, sizeof out, cudaMemcpyDeviceToHost, st);
        if (e == cudaSuccess)
            e = cudaMemcpyAsync(u_out, A.u, sizeof(T) * n * nu, cudaMemcpyDeviceToHost, st);
        if (e == cudaSuccess && err_out)
            e = cudaMemcpyAsync(err_out, A.erriter, sizeof(T) * iterNum, cudaMemcpyDeviceToHost, st);
        if (e == cudaSuccess)
            e = cudaStreamSynchronize(st);
        if (e == cudaSuccess && itNum)
            *itNum = out.it_num;
    }
    if (status == ASETS_OK && e != cudaSuccess) {
        cudaGetLastError();
        status = ASETS_ERR_CUDA;
        set_last_error((std::string("Matlab-semantics solver: ") + cudaGetErrorString(e)).c_str());
    }
    for (void *p : bufs)
        cudaFreeAsync(p, st);
    cudaStreamSynchronize(st);
    return status;
}

// Binary 3D in single precision: one pass per iteration, the 3D iteration
// kernel with the twin's expressions (stencil3d_kernel.cuh, EPI_TWIN), on rows
// padded as it takes them.  160 x 192 x 144: 85 us per iteration against
// 141 with the two passes above (256^3: 215; 528 with the former two passes).

// u, pt and the first gradient source of the padded volume (mt_init, mt_ud)
__global__ void __launch_bounds__(kThreads) mt_init3(const float *cs, const float *ct, float *u, float *pt,
                                                     float *gk, long long cells, int pitch, int nr,
                                                     float cc)
{
    MT_LOOP(cells)
    {
        if ((int)((unsigned int)t % (unsigned int)pitch) >= nr)
            continue;
        const float a = cs[t], b = ct[t], m = mn(a, b);
        const float v = (sub(a, b) >= 0.0f) ? 1.0f : 0.0f;
        u[t] = v;
        pt[t] = m;
        gk[t] = sub(0.0f, add(sub(m, m), dvd(v, cc)));
    }
}

asets_status mt_binary3d_f32(asets_context *ctx, int rows, int cols, int slices, const float *Cs,
                             const float *Ct, const float *alpha, int iterNum, double beta, double cc,
                             double steps, float *u_out, float *err_out, int *itNum)
{
    cudaStream_t st = context_stream(ctx);
    const int sms = context_num_sms(ctx);
    const long long pitch = rows >= 32 ? ((long long)rows + 31) / 32 * 32 : ((long long)rows + 3) / 4 * 4;
    const long long plane = pitch * cols, cells = plane * slices;
    std::vector<void *> bufs;
    cudaError_t e = cudaSuccess;
    auto get = [&](size_t bytes) -> void * {
        void *v = nullptr;
        if (e == cudaSuccess && (e = cudaMallocAsync(&v, bytes, st)) == cudaSuccess)
            bufs.push_back(v);
        return v;
    };
    auto field = [&]() { return static_cast<float *>(get((size_t)cells * sizeof(float))); };
    StencilProblem p;
    memset(&p, 0, sizeof p);
    p.nr = rows;
    p.nc = cols;
    p.ns = slices;
    p.pitch = pitch;
    p.plane = plane;
    p.cells = cells;
    p.flow_labels = p.alpha_labels = p.ct_labels = 1;
    p.src_labels[0] = p.src_labels[1] = p.src_labels[2] = 1;
    float *cs = field(), *ct = field();
    p.alpha = field();
    p.cs = cs;
    p.ct = ct;
    for (int par = 0; par < 2; ++par) {
        for (int k = 0; k < 3; ++k)
            p.b[par][k] = field();
        for (int k = 0; k < 3; ++k)
            p.src[par][k] = field();  // gk, pt, u
    }
    for (int par = 0; par < 2; ++par)
        for (int k = 0; k < 3; ++k)
            p.dst_s[par][k] = p.src[par ^ 1][k];
    int nv = 0;
    const StencilVariant *tab = binary3d_twin_variants(&nv);
    std::vector<const StencilVariant *> vs;
    for (int i = 0; i < nv; ++i)
        vs.push_back(&tab[i]);
    const StencilVariant *v = pick_split3(p, vs.data(), nv, sms);
    ProblemDesc D;
    asets_status status = ASETS_OK;
    IterControl out;
    memset(&out, 0, sizeof out);
    if (e == cudaSuccess) {
        const int r = build_problem_desc(context_encoder(ctx), *v, p, &D);
        if (r) {
            status = ASETS_ERR_CUDA;
            set_last_error("Matlab-semantics solver: cuTensorMapEncodeTiled failed");
        }
    }
    if (e == cudaSuccess && status == ASETS_OK) {
        choose_split3(p, *v, sms, &D);
        const int items = split3_items(p, *v, D);
        IterControl c0;
        memset(&c0, 0, sizeof c0);
        c0.last_iter = -1;
        c0.max_it = iterNum;
        c0.break_lt = 1;
        c0.err_bound = (float)beta;
        c0.denom = 1.0f;
        c0.vol = (double)((long long)rows * cols * slices);
        D.n_items = items;
        D.item_begin = 0;
        D.ctl = static_cast<IterControl *>(get(sizeof(IterControl)));
        D.item_partials = static_cast<double *>(get(sizeof(double) * items));
        D.cvg = static_cast<float *>(get(sizeof(float) * iterNum));
        D.cc = (float)cc;
        D.inv_cc = 1.0f / (float)cc;
        D.inv_cc_l = (float)(1.0 / cc);
        D.steps = (float)steps;
        BatchArgs B;
        ProblemDesc *d_desc = static_cast<ProblemDesc *>(get(sizeof(ProblemDesc)));
        int *map = static_cast<int *>(get(sizeof(int) * items));
        B.probs = d_desc;
        B.item_problem = map;
        B.total_items = items;
        B.queue = static_cast<unsigned int *>(get(4 * sizeof(unsigned int)));
        B.done_count = B.queue + 2;
        B.use_maps(D);
        auto tr = [&](cudaError_t r) {
            if (e == cudaSuccess)
                e = r;
        };
        const size_t w = (size_t)rows * sizeof(float), pw = (size_t)pitch * sizeof(float);
        const size_t h = (size_t)cols * slices;
        if (e == cudaSuccess) {
            // across in one run, then padded (a pitched copy from pageable
            // memory goes row by row); the staging is the second flow buffer
            auto put = [&](float *dst, const float *src, float *stage) {
                tr(cudaMemcpyAsync(pw == w ? dst : stage, src, w * h, cudaMemcpyHostToDevice, st));
                if (pw != w)
                    tr(cudaMemcpy2DAsync(dst, pw, stage, w, w, h, cudaMemcpyDeviceToDevice, st));
            };
            put(ct, Ct, p.b[1][0]);
            put(p.alpha, alpha, p.b[1][1]);
            put(cs, Cs, p.b[1][2]);
            tr(cudaMemcpyAsync(d_desc, &D, sizeof D, cudaMemcpyHostToDevice, st));
            tr(cudaMemcpyAsync(D.ctl, &c0, sizeof c0, cudaMemcpyHostToDevice, st));
            tr(cudaMemsetAsync(map, 0, sizeof(int) * items, st));
            tr(cudaMemsetAsync(B.queue, 0, 4 * sizeof(unsigned int), st));
            tr(cudaMemsetAsync(D.cvg, 0, sizeof(float) * iterNum, st));
            for (int k = 0; k < 3; ++k)
                tr(cudaMemsetAsync(p.b[0][k], 0, (size_t)cells * sizeof(float), st));
        }
        if (e == cudaSuccess) {
            mt_init3<<<mt_grid(cells, sms), kThreads, 0, st>>>(cs, ct, p.src[0][2], p.src[0][1],
                                                               p.src[0][0], cells, (int)pitch, rows,
                                                               (float)cc);
            tr(cudaGetLastError());
            tr(cudaFuncSetAttribute(v->fn, cudaFuncAttributeMaxDynamicSharedMemorySize, v->smem_bytes));
        }
        constexpr int kChunk = 16;
        void *params[] = {&B};
        const dim3 grid((unsigned int)(items < sms ? items : sms));
        for (int i = 0; e == cudaSuccess && i < iterNum && !out.done; i += kChunk) {
            for (int j = i; j < i + kChunk && j < iterNum; ++j)
                tr(cudaLaunchKernel(v->fn, grid, dim3(v->nt), params, v->smem_bytes, st));
            tr(cudaMemcpyAsync(&out, D.ctl, sizeof out, cudaMemcpyDeviceToHost, st));
            tr(cudaStreamSynchronize(st));
        }
        if (e == cudaSuccess && (out.error & DEV_ERR_TIMEOUT)) {
            status = ASETS_ERR_TIMEOUT;
            set_last_error("Matlab-semantics solver: a device-side wait timed out");
        } else if (e == cudaSuccess && out.error) {
            status = ASETS_ERR_CUDA;
            set_last_error("Matlab-semantics solver: an out-of-range access was caught");
        }
        const float *u = p.src[(out.last_iter + 1) & 1][2];
        if (pw != w) {
            tr(cudaMemcpy2DAsync(p.b[0][0], w, u, pw, w, h, cudaMemcpyDeviceToDevice, st));
            u = p.b[0][0];
        }
        tr(cudaMemcpyAsync(u_out, u, w * h, cudaMemcpyDeviceToHost, st));
        if (err_out)
            tr(cudaMemcpyAsync(err_out, D.cvg, sizeof(float) * iterNum, cudaMemcpyDeviceToHost, st));
        tr(cudaStreamSynchronize(st));
        if (itNum)
            *itNum = out.last_iter + 1;
    }
    if (status == ASETS_OK && e != cudaSuccess) {
        cudaGetLastError();
        status = e == cudaErrorMemoryAllocation ? ASETS_ERR_OUT_OF_MEMORY : ASETS_ERR_CUDA;
        set_last_error((std::string("Matlab-semantics solver: ") + cudaGetErrorString(e)).c_str());
    }
    for (void *b : bufs)
        cudaFreeAsync(b, st);
    cudaStreamSynchronize(st);
    return status;
}

// Voxels from which the one-pass form is the faster one (us per iteration, one
// pass against two: 48^3 25.5 / 20.0, 128 x 128 x 10 25.3 / 24.2, 64^3
// 23.5 / 29.3, 128 x 100 x 60 29.7 / 43.0).
constexpr long long kOnePassMin = 200000;
// and rows: its tiles have 64 (4 x 400 x 300 103.6 / 33.1, 8 x 300 x 200 62.2 / 33.4, 16
// x 300 x 100 41.3 / 33.1).
constexpr int kOnePassRows = 24;

template <class T>
asets_status mt_dispatch(int model, int dim, asets_context *ctx, int rows, int cols, int slices,
                         int nlab, const void *Cs, const void *Ct, const void *alpha, int iterNum,
                         double beta, double cc, double steps, void *u, void *err, int *itNum)
{
    if constexpr (sizeof(T) == 4)
        if (model == MT_BINARY && dim == 3 && rows >= kOnePassRows && (long long)rows * cols * slices >= kOnePassMin) {
            const asets_status s =
                mt_binary3d_f32(ctx, rows, cols, slices, static_cast<const float *>(Cs),
                                static_cast<const float *>(Ct), static_cast<const float *>(alpha), iterNum, beta,
                                cc, steps, static_cast<float *>(u), static_cast<float *>(err), itNum);
            if (s != ASETS_ERR_OUT_OF_MEMORY)  // the two passes' rows are not padded
                return s;
        }
#define MT_CASE(M, D)                                                                       \
    if (model == M && dim == D)                                                             \
        return mt_run<T, M, D>(ctx, rows, cols, slices, nlab, Cs, Ct, alpha, iterNum, beta, \
                               cc, steps, u, err, itNum);
    MT_CASE(MT_BINARY, 2)
    MT_CASE(MT_BINARY, 3)
    MT_CASE(MT_POTTS, 2)
    MT_CASE(MT_POTTS, 3)
    MT_CASE(MT_ISHIKAWA, 2)
    MT_CASE(MT_ISHIKAWA, 3)
#undef MT_CASE
    set_last_error("Matlab-semantics solver: bad model or dimension");
    return ASETS_ERR_INVALID_ARG;
}

}  // namespace

extern "C" ASETS_API asets_status asets_matlab_solve(
    asets_context *ctx, int model, int precision, int dim, int rows, int cols, int slices,
    int nlab, const void *Cs, const void *Ct, const void *alpha, int iterNum, double beta,
    double cc, double steps, void *u, void *erriter, int *itNum, float *seconds)
{
    if (!ctx || !Ct || !alpha || !u || iterNum < 1 || rows < 1 || cols < 1 || slices < 1 ||
        (dim != 2 && dim != 3) || (dim == 2 && slices != 1) || (precision != 4 && precision != 8) ||
        (model == MT_BINARY && !Cs) || (model == MT_POTTS && nlab < 1) ||
        (model == MT_ISHIKAWA && nlab < 2) || model < 0 || model > 2) {
        set_last_error("asets_matlab_solve: bad arguments");
        return ASETS_ERR_INVALID_ARG;
    }
    if ((long long)(rows + 1) * (cols + 1) * (slices + 1) * (nlab > 1 ? nlab : 1) >= (1LL << 31)) {
        set_last_error("asets_matlab_solve: volume x labels must stay below 2^31 elements");
        return ASETS_ERR_INVALID_ARG;
    }
    const auto t0 = std::chrono::steady_clock::now();
    int prev = 0;
    cudaGetDevice(&prev);
    cudaSetDevice(context_device(ctx));
    const asets_status s =
        precision == 8 ? mt_dispatch<double>(model, dim, ctx, rows, cols, slices, nlab, Cs, Ct,
                                             alpha, iterNum, beta, cc, steps, u, erriter, itNum)
                       : mt_dispatch<float>(model, dim, ctx, rows, cols, slices, nlab, Cs, Ct,
                                            alpha, iterNum, beta, cc, steps, u, erriter, itNum);
    cudaSetDevice(prev);
    if (seconds)
        *seconds = std::chrono::duration<float>(std::chrono::steady_clock::now() - t0).count();
    return s;
}
