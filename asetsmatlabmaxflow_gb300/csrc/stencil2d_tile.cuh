// Binary 2D iteration on square tiles, for problems too small to keep the
// column sweep of stencil2_kernel.cuh busy.
//
// The sweep kernels walk each (tile, chunk) item plane by plane: on a 256^2
// image a launch has a few dozen items of 8-16 planes each, so the time of
// an iteration is the latency of one item's sweep, not bandwidth.  Here a
// block computes one whole iteration of an R x S tile (rows x stream
// columns) from the old state in phases over a shared frame of
// (R+5) x (S+5) cells (the tile and the iteration's two-cell halo, plus the
// faces beyond it): gk, then the gradient step b', the projection g2, the
// new flows b'' and, on the tile, the divergence and the ps/pt/u update with
// erriter -- the same float expressions, in the same order and with the
// same border masks, as the sweep kernel (EXACT results are bit-identical).
// Old state is read with coalesced loads through L2 (a small problem sits in
// L2), all of a thread's loads in flight at once; out-of-volume cells read
// as 0, the zero-flux border.  Two kernels: one launch per iteration, items
// handed out by the same queue and closed by the same per-item erriter
// partials and ticket as the sweeps; or every iteration in one cooperative
// launch with a grid barrier between iterations (every block resident, each
// taking one or more tiles), which removes the launch and hand-off latency
// that dominates an iteration of a small image.
#pragma once

#include "stencil2_kernel.cuh"

namespace asets {

template <int R, int S>
struct Tile2Geom {
    static constexpr int FR = R + 5;          // frame rows: r0-2 .. r0+R+2
    static constexpr int FC = S + 5;          // frame columns: s0-2 .. s0+S+2
    static constexpr int F = FR * FC;         // floats per frame array
    static constexpr int NARR = 10;           // BR BS PS PT U AL GK BR1 BS1 G2
    static constexpr int smem_bytes() { return NARR * F * 4 + 16; }
};

// A thread's loads of a tile: its frame cells, and Cs/Ct of its tile cells for
// the update.  All are issued before the first is used: one memory round trip.
// State is read through L2 (ld.global.cg): the persistent kernel reads what
// other blocks wrote during the same launch.  `keep`: Cs and Ct, the tile's
// own cells and alpha are those of the iteration before.
template <int R, int S, int NT>
struct Tile2Loads {
    using G = Tile2Geom<R, S>;
    static constexpr int PER = (G::F + NT - 1) / NT;
    static constexpr int PIX = (R * S + NT - 1) / NT;
    float v[6][PER], cs[PIX], ct[PIX];
    bool kept;

    // frame cell k of this thread was loaded (with keep: lies around the tile)
    __device__ static bool wanted(int i, bool keep)
    {
        const int c = i / G::FR, q = i - c * G::FR;
        return i < G::F && !(keep && c >= 2 && c < S + 2 && q >= 2 && q < R + 2);
    }
    __device__ void issue(const ProblemDesc &P, int par, int li, bool keep)
    {
        const int tid = threadIdx.x, nr = P.nr, ns = P.ns;
        const int r0 = (li % P.tiles_r) * R, s0 = (li / P.tiles_r) * S;
        const unsigned int pitch = (unsigned int)P.plane_stride;
        const float *src_br = P.dst_b[par ^ 1][SL_BR], *src_bs = P.dst_b[par ^ 1][SL_BS];
        const float *src_ps = P.dst_s[par ^ 1][0], *src_pt = P.dst_s[par ^ 1][1], *src_u = P.dst_s[par ^ 1][2];
        kept = keep;
        // frame cell (c, q) <-> pixel (r0-2+q, s0-2+c)
#pragma unroll
        for (int k = 0; k < PER; ++k) {
            const int i = tid + k * NT;
            const int c = i / G::FR, q = i - c * G::FR;
            const int r = r0 - 2 + q, s = s0 - 2 + c;
            const bool in = (wanted(i, keep) && r >= 0 && r < nr && s >= 0 && s < ns);
            const unsigned int g = (unsigned int)s * pitch + (unsigned int)r;
            v[0][k] = in ? __ldcg(src_br + g) : 0.f;
            v[1][k] = in ? __ldcg(src_bs + g) : 0.f;
            v[2][k] = in ? __ldcg(src_ps + g) : 0.f;
            v[3][k] = in ? __ldcg(src_pt + g) : 0.f;
            v[4][k] = in ? __ldcg(src_u + g) : 0.f;
            if (!keep)
                v[5][k] = in ? __ldcg(P.alpha + g) : 0.f;
        }
        if (keep)
            return;
#pragma unroll
        for (int k = 0; k < PIX; ++k) {
            const int i = tid + k * NT;
            const int r = r0 + i % R, s = s0 + i / R;
            const bool in = (i < R * S && r < nr && s < ns);
            const unsigned int g = (unsigned int)s * pitch + (unsigned int)r;
            cs[k] = in ? __ldcg(P.cs + g) : 0.f;
            ct[k] = in ? __ldcg(P.ct + g) : 0.f;
        }
    }
    // into the frame arrays (BR BS PS PT U AL); ALL: they were not issued with keep
    template <bool ALL>
    __device__ void store(float *fsm) const
    {
        const bool around = !ALL && kept;
#pragma unroll
        for (int k = 0; k < PER; ++k) {
            const int i = threadIdx.x + k * NT;
            if (wanted(i, around)) {
#pragma unroll
                for (int a = 0; a < 5; ++a)
                    fsm[a * G::F + i] = v[a][k];
                if (!around)
                    fsm[5 * G::F + i] = v[5][k];
            }
        }
    }
};

// One ALM iteration of tile li of problem P from parity par, in the frame
// `fsm` (Tile2Geom::NARR arrays): the loads' arrival, the phases, the stores
// of the new flows and (with KEEP) the state, which stay in the frame as well.
// Returns the thread's share of erriter.
template <int R, int S, int NT, bool EXACT, bool KEEP = false>
__device__ __forceinline__ float tile2_iteration(const ProblemDesc &P, int par, int li, float *fsm,
                                                 const Tile2Loads<R, S, NT> &in)
{
    using G = Tile2Geom<R, S>;
    constexpr int FR = G::FR, F = G::F;
    float *BR = fsm, *BS = fsm + F, *PS = fsm + 2 * F, *PT = fsm + 3 * F, *U = fsm + 4 * F;
    float *AL = fsm + 5 * F, *GK = fsm + 6 * F, *BR1 = fsm + 7 * F, *BS1 = fsm + 8 * F;
    float *G2 = fsm + 9 * F;
    const int tid = threadIdx.x;
    const int nr = P.nr, ns = P.ns;
    const float cc = P.cc, inv_cc = P.inv_cc, steps = P.steps;
    const int r0 = (li % P.tiles_r) * R;
    const int s0 = (li / P.tiles_r) * S;
    const unsigned int pitch = (unsigned int)P.plane_stride;  // one row of Matlab x
    constexpr int PIX = Tile2Loads<R, S, NT>::PIX;
    float erru = 0.0f;
    in.template store<!KEEP>(fsm);
    __syncthreads();

    // gk on rows r0-2 .. r0+R+1, columns s0-2 .. s0+S+1
    for (int i = tid; i < (R + 4) * (S + 4); i += NT) {
        const int c = i / (R + 4), q = i - c * (R + 4);
        const int f = c * FR + q;
        float d = BR[f + 1] - BR[f];
        d = d + BS[f + FR];
        d = d - BS[f];
        GK[f] = d - ((PS[f] - PT[f]) + div_cc<EXACT>(U[f], cc, inv_cc));
    }
    __syncthreads();

    // b'_r on faces r0-1 .. r0+R+1 of columns s0-1 .. s0+S; b'_s on
    // faces s0-1 .. s0+S+1 of rows r0-1 .. r0+R
    for (int i = tid; i < (R + 3) * (S + 2); i += NT) {
        const int c = 1 + i / (R + 3), q = 1 + i % (R + 3);
        const int f = c * FR + q;
        const int r = r0 - 2 + q, s = s0 - 2 + c;
        const bool fr_ok = (r >= 1 && r < nr), s_in = (s >= 0 && s < ns);
        BR1[f] = keep_if<EXACT>(steps * (GK[f] - GK[f - 1]) + BR[f], fr_ok && s_in,
                                fr_ok ? 1.f : 0.f);
    }
    for (int i = tid; i < (R + 2) * (S + 3); i += NT) {
        const int c = 1 + i / (R + 2), q = 1 + i % (R + 2);
        const int f = c * FR + q;
        const int r = r0 - 2 + q, s = s0 - 2 + c;
        const bool inplane = (r >= 0 && r < nr), sb_in = (s >= 1 && s < ns);
        BS1[f] = keep_if<EXACT>(steps * (GK[f] - GK[f - FR]) + BS[f], inplane && sb_in,
                                sb_in ? 1.f : 0.f);
    }
    __syncthreads();

    // g2 on rows r0-1 .. r0+R, columns s0-1 .. s0+S
    for (int i = tid; i < (R + 2) * (S + 2); i += NT) {
        const int c = 1 + i / (R + 2), q = 1 + i % (R + 2);
        const int f = c * FR + q;
        G2[f] = Proj<EXACT>::gk(BS1[f + FR], BS1[f], BR1[f + 1], BR1[f], AL[f]);
    }
    __syncthreads();

    // b''_r on faces r0 .. r0+R of the tile's columns, b''_s on faces
    // s0 .. s0+S of the tile's rows (into the old-flow arrays); the
    // tile's own faces are stored
    float *__restrict__ d_br = P.dst_b[par][SL_BR];
    float *__restrict__ d_bs = P.dst_b[par][SL_BS];
    for (int i = tid; i < (R + 1) * S; i += NT) {
        const int c = 2 + i / (R + 1), q = 2 + i % (R + 1);
        const int f = c * FR + q;
        const int r = r0 - 2 + q, s = s0 - 2 + c;
        const bool fr_ok = (r >= 1 && r < nr), sp_in = (s >= 0 && s < ns);
        const float v = keep_if<EXACT>(((G2[f] + G2[f - 1]) * 0.5f) * BR1[f], fr_ok && sp_in,
                                       fr_ok ? 1.f : 0.f);
        BR[f] = v;
        if (q < R + 2 && r < nr && s < ns)
            d_br[(unsigned int)s * pitch + (unsigned int)r] = v;
    }
    for (int i = tid; i < R * (S + 1); i += NT) {
        const int c = 2 + i / R, q = 2 + i % R;
        const int f = c * FR + q;
        const int r = r0 - 2 + q, s = s0 - 2 + c;
        const bool inplane = (r >= 0 && r < nr), spb_in = (s >= 1 && s < ns);
        const float v = keep_if<EXACT>(((G2[f] + G2[f - FR]) * 0.5f) * BS1[f],
                                       inplane && spb_in, spb_in ? 1.f : 0.f);
        BS[f] = v;
        if (c < S + 2 && r < nr && s < ns)
            d_bs[(unsigned int)s * pitch + (unsigned int)r] = v;
    }
    __syncthreads();

    // the tile: divergence of b'', ps/pt/u, erriter
    float *__restrict__ d_ps = P.dst_s[par][0];
    float *__restrict__ d_pt = P.dst_s[par][1];
    float *__restrict__ d_u = P.dst_s[par][2];
#pragma unroll
    for (int k = 0; k < PIX; ++k) {
        const int i = tid + k * NT;
        const int c = 2 + i / R, q = 2 + i % R;
        const int r = r0 - 2 + q, s = s0 - 2 + c;
        if (i >= R * S || r >= nr || s >= ns)
            continue;
        const int f = c * FR + q;
        float dv = BR[f + 1] - BR[f];
        dv = dv + BS[f + FR];
        dv = dv - BS[f];
        const unsigned int g = (unsigned int)s * pitch + (unsigned int)r;
        const float u = U[f];
        const float ucc = div_cc<EXACT>(u, cc, inv_cc);
        float ps_n = ((PT[f] - ucc) + dv) + inv_cc;
        ps_n = min_sel<EXACT>(ps_n, in.cs[k]);
        float pt_n = (ps_n + ucc) - dv;
        pt_n = min_sel<EXACT>(pt_n, in.ct[k]);
        const float e = cc * ((pt_n + dv) - ps_n);
        erru += abs_ref(e);
        d_ps[g] = ps_n;
        d_pt[g] = pt_n;
        d_u[g] = u - e;
        if (KEEP) {
            PS[f] = ps_n;
            PT[f] = pt_n;
            U[f] = u - e;
        }
    }
    __syncthreads();  // the frame is reused by the next item or iteration
    return erru;
}

template <int R, int S, int NT, bool EXACT, int MINB>
__global__ void __launch_bounds__(NT, MINB) stencil2d_tile_kernel(const __grid_constant__ BatchArgs B)
{
    extern __shared__ __align__(16) float fsm[];
    __shared__ double s_red[NT / 32];
    __shared__ int s_is_last;
    __shared__ int s_item;
    __shared__ int s_iter;
    const int tid = threadIdx.x;

    while (true) {
        if (tid == 0) {
            const int itm = (int)atomicAdd(&B.queue[0], 1u);
            int iter = -1;
            if (itm < B.total_items) {
                const IterControl *c = B.probs[B.item_problem[itm]].ctl;
                iter = *(const volatile int *)&c->done ? -1 : *(const volatile int *)&c->iter;
            }
            s_item = itm;
            s_iter = iter;
        }
        __syncthreads();
        const int item = s_item;
        const int it = s_iter;
        __syncthreads();  // s_item/s_iter are rewritten by the next fetch
        if (item >= B.total_items)
            break;
        if (it < 0)
            continue;  // the problem has converged
        const ProblemDesc &P = B.probs[B.item_problem[item]];
        const int li = item - P.item_begin;
        Tile2Loads<R, S, NT> in;
        in.issue(P, it & 1, li, false);
        const float erru = tile2_iteration<R, S, NT, EXACT>(P, it & 1, li, fsm, in);
        finish_item<NT>(erru, P, li, it, B.done_count, s_red, &s_is_last);
    }

    // the last block to leave re-arms the queue for the next launch
    if (tid == 0) {
        __threadfence();
        if (atomicAdd(&B.queue[1], 1u) == gridDim.x - 1) {
            B.queue[0] = 0;
            B.queue[1] = 0;
            __threadfence();
        }
    }
}

// Every iteration of one problem in one cooperative launch: block b takes
// tiles b, b + grid, ... of every iteration (`iteration(it, tile)` returns
// the thread's erriter share); after each iteration the blocks meet at a grid barrier (an arrival
// counter, zeroed before the launch; each wait bounded by time, a timeout
// sets DEV_ERR_TIMEOUT and ends the solve), then every block sums the
// blocks' erriter partials in the order finish_item uses for items, so all
// take the same stopping decision; block 0 records cvg, itNum and the
// control block as finish_item does.  The launch and per-iteration hand-off of the
// one-launch-per-iteration form (queue, ticket, kernel boundary) is replaced
// by one barrier.  Partials alternate between two halves of item_partials by
// iteration parity.
//
// `load(it, tile, keep)` starts a tile's loads and `iteration` completes them.
// The loads of a block's first tile start as soon as the barrier has opened,
// before the stopping decision; where every block has one tile, its own cells
// stay on chip (keep) and only their surroundings are loaded.  An iteration is
// a chain of latencies: of 24,000 cycles for a Potts tile with four labels,
// 8,500 were its phases, 4,400 the block's sum in double, 4,200 the decision
// after the loads' issue and the rest the barrier; with the sum in pairs, the
// decision beside the loads and its partials in flight together, 301 x 170
// with four labels takes 8.7 us an iteration (11.9 before), binary 256 x 256
// 5.5 (6.3).
//
// TILES: one tile a block, several, or (TILES_ANY) whichever the launch has.  The
// binary kernels are compiled for each apart: with both loops in one kernel
// several tiles a block took 2 to 4 % longer (EXACT 1100 x 1100 38.6 us an iteration
// against 37.6).
enum Tiles { TILES_ONE, TILES_MANY, TILES_ANY };
template <int NT, int TILES, class Load, class Iteration>
__device__ __forceinline__ void tile_solve_loop(const ProblemDesc &P, unsigned int *arrivals,
                                                double *s_red, int *s_stop, Load load, Iteration iteration)
{
    const int tid = threadIdx.x;
    IterControl *ctl = P.ctl;
    const int nb = (int)gridDim.x;   // at most one block per tile
    const int li = (int)blockIdx.x;
    if (*(volatile int *)&ctl->done)
        return;
    int it = *(volatile int *)&ctl->iter;
    const int max_it = ctl->max_it;
    const int break_lt = ctl->break_lt;
    const float err_bound = ctl->err_bound, denom = ctl->denom;
    const bool one = TILES == TILES_ANY ? P.n_items <= nb : TILES == TILES_ONE;
    if (TILES != TILES_MANY)
        load(it, li, false);
    for (unsigned int gen = 1;; ++gen) {
        float erru = TILES != TILES_MANY ? iteration(it, li) : 0.0f;
        if (TILES != TILES_ONE)
            for (int tile = TILES == TILES_MANY ? li : li + nb; tile < P.n_items; tile += nb) {
                load(it, tile, false);
                erru += iteration(it, tile);
            }
        const double part = block_sum<NT>(erru, s_red);
        if (tid == 0) {
            P.item_partials[(it & 1) * nb + li] = part;
            __threadfence();
            atomicAdd(arrivals, 1u);
            // grid barrier: every block's state and partial of iteration it
            const unsigned int target = gen * (unsigned int)nb;
            int stop = 0;
            if (*(volatile unsigned int *)arrivals < target) {
                const unsigned long long t0 = global_timer_ns();
                while (*(volatile unsigned int *)arrivals < target) {
                    if (global_timer_ns() - t0 > kWaitBudgetNs) {
                        atomicOr(&ctl->error, DEV_ERR_TIMEOUT);
                        stop = 2;
                        break;
                    }
                }
            }
            __threadfence();
            *s_stop = stop;
        }
        __syncthreads();
        if (*s_stop == 2)
            break;  // a block did not arrive
        // the loads of the next iteration cover warp 0's decision
        if (TILES != TILES_MANY)
            load(it + 1, li, one);
        if (tid < 32) {
            double acc = lane_partials(P.item_partials + (it & 1) * nb, nb);
#pragma unroll
            for (int o = 16; o > 0; o >>= 1)
                acc += __shfl_xor_sync(0xffffffffu, acc, o);
            if (tid == 0) {
                // cvg[i] = total_err / (float)N, total_err a float (runMaxFlow)
                const float c = __fdiv_rn((float)acc, denom);
                const bool conv = break_lt ? (c < err_bound) : (c <= err_bound);
                const int done = (conv || it + 1 >= max_it) ? 1 : 0;
                if (li == 0) {
                    P.cvg[it] = c;
                    ctl->last_iter = it;
                    ctl->iter = it + 1;
                    if (done) {
                        ctl->it_num = conv ? it : max_it;
                        ctl->done = 1;
                    }
                }
                *s_stop = done;
            }
        }
        __syncthreads();
        if (*s_stop)
            break;
        ++it;
    }
}

template <int R, int S, int NT, bool EXACT, int MINB, int TILES>
__global__ void __launch_bounds__(NT, MINB)
    stencil2d_tile_persistent_kernel(const __grid_constant__ BatchArgs B)
{
    extern __shared__ __align__(16) float fsm[];
    __shared__ double s_red[NT / 32];
    __shared__ int s_stop;
    const ProblemDesc &P = B.probs[0];
    Tile2Loads<R, S, NT> in;
    tile_solve_loop<NT, TILES>(
        P, B.queue, s_red, &s_stop,
        [&](int it, int tile, bool keep) { in.issue(P, it & 1, tile, keep); },
        [&](int it, int tile) {
            return tile2_iteration<R, S, NT, EXACT, TILES == TILES_ONE>(P, it & 1, tile, fsm, in);
        });
}

}  // namespace asets
