// Fused 3D ALM iteration kernel with a carried gradient source: one launch =
// one iteration of the flows of every label and, for the binary model, of
// ps/pt/u and erriter.
//
// It fuses, per label, the reference's updateP1, updatePX/PY/PZ, projStep,
// updateBX/BY/BZ and divergence sweeps (maxflow/asetsBinaryMF3D_mex.c:166-180)
// and, for the binary model, updateDIVPSPTU and the erriter sum (:398-437).
//
// Carried source.  The gradient step reads gk = div b - ((ps - pt) + u/cc)
// two cells around every face.  The iteration that forms ps, pt and u of a
// cell has its divergence at hand, so it stores gk there and then (for the
// labelled models the label kernel does), the same float expression on the
// same operands as the reference forms it at the start of the next iteration.
// A step then needs no divergence of the old flows on the halo, no block
// barrier to exchange gk, and five halo boxes (gk, three flows, alpha)
// instead of seven; ps is not read by any later iteration and is not stored
// (carry3d.cu forms it on request from the state before the last iteration).
//
// Geometry.  Rows r (Matlab y, contiguous), columns c (Matlab x) and a
// stream axis s (z).  A tile is 32*CELLS rows x TC columns; main warp w is
// column c0-1+w, a lane owns CELLS adjacent rows of it for the whole sweep
// along s.  The projection factors one cell around the tile are needed too:
// columns -1 and TC are main warps of their own, rows -1 and 32*CELLS of the
// TC tile columns are the lanes of one more warp (the tile needs no corner).
// So a warp's rows are all tile rows and row counts of 32*CELLS multiples
// leave no ragged tile.  Step s computes
//   Y: b'(s) from gk(s); projection g2(s-1); b''_s(s-1)
//   Z: b''_r, b''_c of plane s-1; ps/pt/u and gk (or div) of plane s-2
// with one block barrier per step, for the factors of the neighbouring
// columns (a plane double-buffered in shared memory); row neighbours come
// from the thread itself or one warp shuffle.  Old-state planes come through
// a ring of 4D TMA tiled loads, one mbarrier per stage; a stage holds the
// halo boxes of plane s and, for the binary model, the tile boxes of plane
// s-2.  All of it is read before the step's barrier, after which the slot is
// refilled.  Out-of-grid elements load as 0: the reference's zero-flux border.
//
// Cold start (EPI_COLD, fast binary).  From the reference's own initial state
// on, u is not zero only where pt = Ct: with p = (ps' + u/cc) - dv and
// pt' = min(p, Ct), u' = cc*(p - pt').  So one float holds both (cold_v), and
// the rounding noise that the subtraction leaves in u where pt < Ct is a zero.
// A start from given pt and u need not satisfy that and keeps both
// (EPI_BINARY), as do EXACT, for the reference's own roundings, and inputs
// out of the joint state's range (kColdInputLimit, cold_cc).
//
// EPI_TWIN: the binary 3D Matlab twin in single precision (mtwin.cu), whose
// expressions differ in order; its erriter is summed to double precision.
//
// Bound: HBM.  Binary 52 B per voxel and iteration (gk, three flows, v in and
// out; alpha, Cs, Ct in), 64 B with pt and u apart; labelled models 36 B per
// label.
//
// Measured (binary 256^3, us per iteration, beside the form that recomputed gk
// from seven halo boxes with two barriers per step): fast 142 (3.5 TB/s on
// the old form's 60 B, 6.1 on the 52 B) against 206, EXACT 253 against 390;
// the flow pass and label kernel of Potts 192^3 L = 4: 270 against 378.
// Three stages, not the five or six that fit: the ring then holds what the
// blocks need and they stay near one another in s, so that the halos are
// found in L2 (six stages: 170 us, 7% more DRAM reads).
//
// Work split: units (label, tile) times chunks of the stream axis, in two
// parts with their own chunk counts (choose_split3), chunk-major so that
// blocks running together hold neighbouring tiles at the same planes; an
// atomic queue hands the items out.  erriter and the stopping rule as in
// stencil2_kernel.cuh.
#pragma once

#include "stencil2_kernel.cuh"

namespace asets {

template <int TC_, int CELLS, int EPI>
struct Geom3 {
    static_assert(CELLS == 1 || CELLS == 2, "one or two cells per lane");
    static_assert(TC_ >= 1 && TC_ <= 16, "the halo rows' warp holds two lanes per tile column");
    static constexpr int TC = TC_;
    static constexpr int TR = 32 * CELLS;
    static constexpr int NW = TC + 2;              // main warps: columns -1 .. TC
    static constexpr int NT = 32 * (NW + 1);       // and the halo rows' warp
    static constexpr int LR = TR + 8;              // box rows r0-4 .. r0+TR+3
    static constexpr int COLS_G = TC + 4;          // gk: columns -2 .. TC+1
    static constexpr int COLS_BC = TC + 3;         // column faces: -1 .. TC+1
    static constexpr int COLS = TC + 2;            // the others: -1 .. TC
    static constexpr int NTILE = (EPI == EPI_BINARY || EPI == EPI_TWIN) ? 4 : (EPI == EPI_COLD ? 3 : 0);
    static constexpr int align128(int b) { return (b + 127) & ~127; }
    // float offsets of the boxes in a stage
    static constexpr int OFF_G = 0;
    static constexpr int OFF_BC = OFF_G + align128(LR * COLS_G * 4) / 4;
    static constexpr int OFF_BR = OFF_BC + align128(LR * COLS_BC * 4) / 4;
    static constexpr int OFF_BS = OFF_BR + align128(LR * COLS * 4) / 4;
    static constexpr int OFF_AL = OFF_BS + align128(LR * COLS * 4) / 4;
    static constexpr int OFF_T0 = OFF_AL + align128(LR * COLS * 4) / 4;
    static constexpr int TSZ = align128(TR * TC * 4) / 4;
    static constexpr int stage_bytes() { return (OFF_T0 + NTILE * TSZ) * 4; }
    static constexpr int tx_bytes()
    {
        return 4 * (LR * (COLS_G + COLS_BC + 3 * COLS) + NTILE * TR * TC);
    }
    // factor plane: row -1 at float 1 of a column, rows 0.. from float 2
    static constexpr int GP = TR + 4;
    static constexpr int plane_floats() { return NW * GP; }
    static constexpr int smem_bytes(int nstage)
    {
        // stages | two factor planes | mbarriers | alignment slack
        return nstage * stage_bytes() + 2 * align128(plane_floats() * 4) + nstage * 8 + 128;
    }
};

// Projection factor of a cell as the faces use it: the fast path halves it
// here, once per cell instead of once per face (exact: a power of two).
template <bool EXACT>
__device__ __forceinline__ float proj_half(float f0, float f1, float f2, float f3, float f4, float f5,
                                           float alpha)
{
    const float g = Proj<EXACT>::gk(f0, f1, f2, f3, f4, f5, alpha);
    return EXACT ? g : 0.5f * g;
}
// mean of the factors of a face's two cells
template <bool EXACT>
__device__ __forceinline__ float face_mean(float g, float g_nb)
{
    return EXACT ? (g + g_nb) * 0.5f : g + g_nb;
}

// Store of a lane's cells at element offset `off`.  A pair is stored whole
// where its first row is in the volume: with an odd row count the second
// value falls into the row's padding, which nothing reads.
template <int C>
__device__ __forceinline__ void st_rows(float *__restrict__ base, unsigned int off, const float (&v)[C],
                                        bool ok, const ProblemDesc &P)
{
    if (!ok)
        return;
#ifdef ASETS_BOUNDS_CHECK
    if ((long long)off + C - 1 >= P.dst_elems) {
        atomicOr(&P.ctl->error, DEV_ERR_BOUNDS);
        return;
    }
#endif
    st_cells<C>(base + off, v);
}

// gradient step of a face: b + steps*d, zero on a border face (EXACT by the
// reference's select, fast by a zero step: the stored border flow is zero)
template <bool EXACT>
__device__ __forceinline__ float face_step(float b, float d, float steps, bool ok, float steps_ok)
{
    if constexpr (EXACT)
        return ok ? steps * d + b : 0.0f;
    else
        return steps_ok * d + b;
}

// Projection factor in the Matlab twins' order and precision (mtwin.cu):
// lower and upper faces along columns, rows, slices; 1/1 is exactly 1, so no
// division below alpha, and no root where a sum of squares with a margin over
// all roundings is.
__device__ __forceinline__ float proj_twin(float a, float b, float d, float e, float p, float q,
                                           float al)
{
    float m = __fmul_rn(a, a);
    m = __fmaf_rn(b, b, m);
    m = __fmaf_rn(d, d, m);
    m = __fmaf_rn(e, e, m);
    m = __fmaf_rn(p, p, m);
    m = __fmaf_rn(q, q, m);
    if (al > 0x1p-40f && m * (0.5f * (1.0f + 0x1p-18f)) < al * al)
        return 1.0f;
    float s = __fadd_rn(__fmul_rn(a, a), __fmul_rn(b, b));
    s = __fadd_rn(s, __fmul_rn(d, d));
    s = __fadd_rn(s, __fmul_rn(e, e));
    s = __fadd_rn(s, __fmul_rn(p, p));
    s = __fadd_rn(s, __fmul_rn(q, q));
    const float g = __fsqrt_rn(__fmul_rn(s, 0.5f));
    return (g <= al) ? 1.0f : __fdiv_rn(1.0f, __fdiv_rn(g, al));
}

// Matlab's min(a, b); a NaN a is kept.
__device__ __forceinline__ float min_twin(float a, float b) { return (a <= b || a != a) ? a : b; }

template <int TC, int CELLS, int NSTAGE, int EPI, bool EXACT>
__global__ void __launch_bounds__(Geom3<TC, CELLS, EPI>::NT, 1)
    stencil3d_kernel(const __grid_constant__ BatchArgs B)
{
    using G = Geom3<TC, CELLS, EPI>;
    constexpr int NT = G::NT, C = CELLS, LR = G::LR, TR = G::TR;
    constexpr bool BIN = (EPI == EPI_BINARY || EPI == EPI_COLD || EPI == EPI_TWIN);
    constexpr bool TWIN = (EPI == EPI_TWIN);
    static_assert(!TWIN || EXACT, "the twins' float operations are IEEE ones");

    extern __shared__ __align__(128) unsigned char smem_raw[];
    __shared__ int s_abort;
    __shared__ double s_red[NT / 32];
    __shared__ int s_is_last;
    __shared__ int s_item, s_iter, s_maps;

    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;

    unsigned char *smem = smem_align128(smem_raw);
    constexpr int SF = G::stage_bytes() / 4;
    float *stages = reinterpret_cast<float *>(smem);
    float *planes = stages + NSTAGE * SF;
    constexpr int PF = G::align128(G::plane_floats() * 4) / 4;
    uint64_t *bars = reinterpret_cast<uint64_t *>(planes + 2 * PF);

    if (tid == 0) {
        s_abort = 0;
        s_maps = -1;
        for (int i = 0; i < NSTAGE; ++i)
            mbar_init(&bars[i], 1);
        mbar_fence_init();
    }
    __syncthreads();

    // tile boxes of a stage: pt, u, Cs, Ct; EPI_COLD: v (in the place of pt), Cs, Ct
    auto tile_slot = [](int ts) { return EPI == EPI_COLD && ts > 0 ? ts + 1 : ts; };
    // main warps: rows row .. row+C-1 of column w-1; the halo rows' warp:
    // row -1 or TR of a tile column (lanes past the last repeat the first)
    const bool main_w = (w < G::NW);
    const int hl = (lane < 2 * TC) ? lane : 0;
    const int hrow = (hl < TC) ? -1 : TR;
    const int row = main_w ? C * lane : hrow;
    const int col = main_w ? w - 1 : hl % TC;                  // relative to c0
    const int bi = (col + 1) * LR + 4 + row;                   // index in the COLS boxes
    const int gi = (col + 1) * G::GP + 2 + row;                // index in a factor plane
    const bool tile_col = main_w && w >= 1 && w <= TC;
    const int ti = row + col * TR;                             // index in the tile boxes
    // the thread that issues the TMA loads: its warp has no work in Z
    const bool producer = (tid == NT - 32), producer_warp = (tid >= NT - 32);

    constexpr unsigned int kHaloMaps = kHaloMaps2D & ~(1u << SL_S1 | 1u << SL_S2) | 1u << SL_BC;
    constexpr unsigned int kTileMaps =
        !BIN ? 0u : EPI == EPI_COLD ? kTileMapsBinary & ~(1u << TS_S2) : kTileMapsBinary;
    int st = 0;        // ring slot of the next stage to read
    uint32_t ph = 0;   // and its mbarrier phase
    bool aborted = false;

    while (!aborted) {
        // thread 0 takes the next item and reads its problem's iteration
        // state once for the whole block
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
        if (producer_warp && it >= 0)
            tensormaps_acquire<kHaloMaps, kTileMaps>(B, item, it & 1, &s_maps);
        __syncthreads();  // s_item/s_iter are rewritten by the next fetch
        if (item >= B.total_items)
            break;
        if (it < 0)
            continue;  // the problem has converged
        const ProblemDesc &P = B.probs[B.item_problem[item]];
        IterControl *ctl = P.ctl;
        const int par = it & 1;
        const CUtensorMap *hmaps = tensormaps(B, P).halo[par];
        const CUtensorMap *tmaps = tensormaps(B, P).tile[par];
        const int nr = P.nr, nc = P.nc, ns = P.ns;
        const float cc = P.cc, inv_cc = P.inv_cc, steps = P.steps;
        const int tiles = P.tiles_r * P.tiles_c;
        const int li = item - P.item_begin;
        // first part: units_a units in zchunks_a chunks; then the others in zchunks
        const int items_a = P.units_a * P.zchunks_a;
        const bool part_a = li < items_a;
        const int part_li = part_a ? li : li - items_a;
        const int part_units = part_a ? P.units_a : tiles * P.nlab_items - P.units_a;
        const int chunks = part_a ? P.zchunks_a : P.zchunks;
        const int chunk = part_li / part_units;
        const int unit = part_li % part_units + (part_a ? 0 : P.units_a);
        const int k = unit / tiles;
        const int tile = unit % tiles;
        const int s_begin = (int)((long long)ns * chunk / chunks);
        const int s_end = (int)((long long)ns * (chunk + 1) / chunks);
        float erru = 0.0f;
        FloatPair errp;  // the twins sum erriter in double
        const int r0 = (tile % P.tiles_r) * TR;
        const int c0 = (tile / P.tiles_r) * TC;
        const int n_steps = s_end - s_begin + 4;
        const int p_first = s_begin - 2;
        const long long lab_off = (long long)k * P.label_stride;

        auto issue_load = [&](int j, int slot) {
            const int plane = p_first + j;
            float *S = stages + slot * SF;
            uint64_t *bar = &bars[slot];
            mbar_arrive_expect_tx(bar, G::tx_bytes());
            tma_load_4d(S + G::OFF_G, &hmaps[SL_S0], r0 - 4, c0 - 2, plane, k, bar);
            tma_load_4d(S + G::OFF_BC, &hmaps[SL_BC], r0 - 4, c0 - 1, plane, k, bar);
            tma_load_4d(S + G::OFF_BR, &hmaps[SL_BR], r0 - 4, c0 - 1, plane, k, bar);
            tma_load_4d(S + G::OFF_BS, &hmaps[SL_BS], r0 - 4, c0 - 1, plane, k, bar);
            tma_load_4d(S + G::OFF_AL, &hmaps[SL_ALPHA], r0 - 4, c0 - 1, plane, k, bar);
#pragma unroll
            for (int ts = 0; ts < G::NTILE; ++ts)
                tma_load_4d(S + G::OFF_T0 + ts * G::TSZ, &tmaps[tile_slot(ts)], r0, c0, plane - 2, 0, bar);
        };
        if (producer)
            for (int j = 0, q = st; j < NSTAGE && j < n_steps; ++j, q = (q + 1 == NSTAGE) ? 0 : q + 1)
                issue_load(j, q);

        // this thread's cells and border masks
        const int r = r0 + row;
        const int c = c0 + col;
        const bool in_c = (c >= 0 && c < nc);
        const bool is_tile = tile_col && r < nr && in_c;
        bool fr_ok[C], in_r[C];
        float st_r[C];
#pragma unroll
        for (int j = 0; j < C; ++j) {
            const int rj = r + j;
            in_r[j] = (rj >= 0 && rj < nr);
            fr_ok[j] = (rj >= 1 && rj < nr && in_c);             // row face rj
            st_r[j] = fr_ok[j] ? steps : 0.f;
        }
        const int rd = r + (main_w ? C : 1);                                    // the row below the last cell
        const bool frd_ok = (rd >= 1 && rd < nr && in_c);
        const bool fc_ok = (c >= 1 && c < nc), fc1_ok = (c + 1 >= 1 && c + 1 < nc);
        const float st_rd = frd_ok ? steps : 0.f;
        const float st_c = fc_ok ? steps : 0.f, st_c1 = fc1_ok ? steps : 0.f;
        // element offsets fit 32 bits: solves are limited to 2^31 - 1 voxel-labels
        const unsigned int col_off = (unsigned int)(lab_off + (long long)c * P.pitch + r);
        const unsigned int plane_stride = (unsigned int)P.plane_stride;
        // of plane s-1 at the current step
        unsigned int o_sp = col_off + (unsigned int)(p_first - 1) * plane_stride;
        // reads bi-1 .. bi+C in the gk box (a column either side) and the row
        // faces, bi .. bi+C-1 elsewhere; tile boxes ti ..; factor planes gi-1 .. gi+C
        check_index(bi - 1, LR * G::COLS, P);
        check_index(bi + C, LR * G::COLS, P);
        check_index(bi + 2 * LR + C, LR * G::COLS_G, P);
        check_index(bi + LR + C - 1, LR * G::COLS_BC, P);
        if (is_tile)
            check_index(ti + C - 1, TR * TC, P);
        check_index(gi - 1, G::plane_floats(), P);
        check_index(gi + C, G::plane_floats(), P);
        float *__restrict__ d_bs = P.dst_b[par][SL_BS];
        float *__restrict__ d_br = P.dst_b[par][SL_BR];
        float *__restrict__ d_bc = P.dst_b[par][SL_BC];
        float *__restrict__ d_s0 = P.dst_s[par][0];
        float *__restrict__ d_s1 = P.dst_s[par][1];
        float *__restrict__ d_s2 = P.dst_s[par][2];

        // carried from the previous step: gk, the faces b' of its plane
        // (bcr: the next column's, brd: the row's below the last cell)
        float gkprev[C], bsprev[C], g2prev[C], alpha_prev[C], br_prev[C], bc_prev[C], bcr_prev[C];
        float brd_prev = 0.f, bss_cur[C], bss_old[C], dvp[C];
#pragma unroll
        for (int j = 0; j < C; ++j) {
            gkprev[j] = bsprev[j] = br_prev[j] = bc_prev[j] = bcr_prev[j] = 0.f;
            bss_cur[j] = bss_old[j] = dvp[j] = 0.f;
            g2prev[j] = alpha_prev[j] = 1.f;
        }

        // A wait gave up: drain the loads of this item from step `first` up
        // to `issued` (bounded), record the error and leave the item.
        auto abort_item = [&](int first, int issued) {
            if (producer) {
                s_abort = 0;
                int q = st;
                uint32_t p = ph;
                for (int j = first; j < issued; ++j) {
                    mbar_wait_bounded(&bars[q], p, &s_abort);
                    if (++q == NSTAGE) {
                        q = 0;
                        p ^= 1;
                    }
                }
                atomicOr(&ctl->error, DEV_ERR_TIMEOUT);
            }
            __syncthreads();
        };

#pragma unroll 1
        for (int t = 0; t < n_steps && !aborted; ++t) {
            const int s = p_first + t;
            // every thread waits on the mbarrier of the stage it reads, which
            // also makes the stage's data visible to it; a timeout is acted
            // on at the block barrier
            const bool wait_ok = mbar_wait_bounded(&bars[st], ph, &s_abort);
            const bool sb_in = (s >= 1 && s < ns);          // stream face s is interior
            const bool spb_in = (s - 1 >= 1 && s - 1 < ns);
            const bool s_in = (s >= 0 && s < ns), sp_in = (s - 1 >= 0 && s - 1 < ns);
            const float st_s = sb_in ? steps : 0.f;
            const float *S = stages + st * SF + bi;
            float *G2 = planes + (t & 1) * PF + gi;

            // ---- Y: faces b'(s), projection g2(s-1), stream faces b''(s-1)
            float gk[C], gl[C], gr[C], br[C], bc[C], bcr[C], bs[C], al[C], g2[C], brd, gup;
            float tv[G::NTILE > 0 ? G::NTILE : 1][C];
            if (main_w) {
            ld_cells<C>(S + G::OFF_G + LR, gk);
            ld_cells<C>(S + G::OFF_G, gl);
            ld_cells<C>(S + G::OFF_G + 2 * LR, gr);
            ld_cells<C>(S + G::OFF_BC, bc);
            ld_cells<C>(S + G::OFF_BC + LR, bcr);
            ld_cells<C>(S + G::OFF_BR, br);
            ld_cells<C>(S + G::OFF_BS, bs);
            ld_cells<C>(S + G::OFF_AL, al);
            gup = __shfl_up_sync(0xffffffffu, gk[C - 1], 1);
            if (lane == 0)
                gup = S[G::OFF_G + LR - 1];
#pragma unroll
            for (int j = 0; j < C; ++j) {
                br[j] = face_step<EXACT>(br[j], gk[j] - (j ? gk[j - 1] : gup), steps, fr_ok[j] && s_in,
                                         st_r[j]);
                bc[j] = face_step<EXACT>(bc[j], gk[j] - gl[j], steps, fc_ok && in_r[j] && s_in, st_c);
                bcr[j] = face_step<EXACT>(bcr[j], gr[j] - gk[j], steps, fc1_ok && in_r[j] && s_in, st_c1);
                bs[j] = face_step<EXACT>(bs[j], gk[j] - gkprev[j], steps, in_r[j] && in_c && sb_in, st_s);
            }
            brd = __shfl_down_sync(0xffffffffu, br[0], 1);
            if (lane == 31)
                brd = face_step<EXACT>(S[G::OFF_BR + C], S[G::OFF_G + LR + C] - gk[C - 1], steps,
                                       frd_ok && s_in, st_rd);
            if (tile_col) {
                const float *T = stages + st * SF + G::OFF_T0 + ti;
#pragma unroll
                for (int ts = 0; ts < G::NTILE; ++ts)
                    ld_cells<C>(T + ts * G::TSZ, tv[ts]);
            }
            } else {
                gk[0] = S[G::OFF_G + LR];
                br[0] = face_step<EXACT>(S[G::OFF_BR], gk[0] - S[G::OFF_G + LR - 1], steps,
                                         fr_ok[0] && s_in, st_r[0]);
                brd = face_step<EXACT>(S[G::OFF_BR + 1], S[G::OFF_G + LR + 1] - gk[0], steps,
                                       frd_ok && s_in, st_rd);
                bc[0] = face_step<EXACT>(S[G::OFF_BC], gk[0] - S[G::OFF_G], steps,
                                         fc_ok && in_r[0] && s_in, st_c);
                bcr[0] = face_step<EXACT>(S[G::OFF_BC + LR], S[G::OFF_G + 2 * LR] - gk[0], steps,
                                          fc1_ok && in_r[0] && s_in, st_c1);
                bs[0] = face_step<EXACT>(S[G::OFF_BS], gk[0] - gkprev[0], steps,
                                         in_r[0] && in_c && sb_in, st_s);
                al[0] = S[G::OFF_AL];
#pragma unroll
                for (int j = 1; j < C; ++j)
                    gk[j] = br[j] = bc[j] = bcr[j] = bs[j] = al[j] = 0.f;
            }
#pragma unroll
            for (int j = 0; j < C; ++j) {
                if (j > 0 && !main_w)
                    break;
                const float dn = (j + 1 < C && main_w) ? br_prev[j + 1 < C ? j + 1 : j] : brd_prev;
                if constexpr (TWIN)
                    g2[j] = proj_twin(bc_prev[j], bcr_prev[j], br_prev[j], dn, bsprev[j], bs[j],
                                      alpha_prev[j]);
                else
                    g2[j] = proj_half<EXACT>(bcr_prev[j], bc_prev[j], dn, br_prev[j], bs[j], bsprev[j],
                                             alpha_prev[j]);
            }
            if (main_w)
                st_cells<C>(G2, g2);
            else
                G2[0] = g2[0];
            const int sp = s - 1;
            if (tile_col) {
                float bssn[C];
#pragma unroll
                for (int j = 0; j < C; ++j) {
                    bssn[j] = face_mean<EXACT>(g2[j], g2prev[j]) * bsprev[j];
                    if (EXACT && !(in_r[j] && in_c && spb_in))
                        bssn[j] = 0.f;
                }
                if (sp >= s_begin && sp < s_end)
                    st_rows<C>(d_bs, o_sp, bssn, is_tile, P);
#pragma unroll
                for (int j = 0; j < C; ++j) {
                    bss_old[j] = bss_cur[j];
                    bss_cur[j] = bssn[j];
                    g2prev[j] = g2[j];
                }
            }
#pragma unroll
            for (int j = 0; j < C; ++j) {
                gkprev[j] = gk[j];
                bsprev[j] = bs[j];
                alpha_prev[j] = al[j];
            }
            if (__syncthreads_or(!wait_ok)) {
                aborted = true;
                // loads issued: the prologue, then one per earlier step
                abort_item(t, min(n_steps, t + NSTAGE));
                break;
            }
            // every read of this stage is done: refill its slot
            if (producer && t + NSTAGE < n_steps)
                issue_load(t + NSTAGE, st);
            if (++st == NSTAGE) {
                st = 0;
                ph ^= 1;
            }

            // ---- Z: row/column faces of plane s-1 and the output of plane s-2
            if (tile_col) {
                float g2l[C], g2r[C], brr[C], bcc[C], dn[C];
                ld_cells<C>(G2 - G::GP, g2l);
                ld_cells<C>(G2 + G::GP, g2r);
                float g2u = __shfl_up_sync(0xffffffffu, g2[C - 1], 1);
                if (lane == 0)
                    g2u = G2[-1];
#pragma unroll
                for (int j = 0; j < C; ++j) {
                    brr[j] = face_mean<EXACT>(g2[j], (j ? g2[j - 1] : g2u)) * br_prev[j];
                    if (EXACT && !(fr_ok[j] && sp_in))
                        brr[j] = 0.f;
                }
                float brr_dn = __shfl_down_sync(0xffffffffu, brr[0], 1);
                if (lane == 31) {
                    brr_dn = face_mean<EXACT>(G2[C], g2[C - 1]) * brd_prev;
                    if (EXACT && !(frd_ok && sp_in))
                        brr_dn = 0.f;
                }
#pragma unroll
                for (int j = 0; j < C; ++j) {
                    const float brr1 = j + 1 < C ? brr[j + 1 < C ? j + 1 : j] : brr_dn;
                    bcc[j] = face_mean<EXACT>(g2[j], g2l[j]) * bc_prev[j];
                    float bcc1 = face_mean<EXACT>(g2r[j], g2[j]) * bcr_prev[j];
                    if (EXACT) {
                        if (!(fc_ok && in_r[j] && sp_in))
                            bcc[j] = 0.f;
                        if (!(fc1_ok && in_r[j] && sp_in))
                            bcc1 = 0.f;
                    }
                    // the reference adds rows, then columns; the twins the other way
                    if constexpr (TWIN)
                        dn[j] = ((bcc1 - bcc[j]) + brr1) - brr[j];
                    else
                        dn[j] = ((brr1 - brr[j]) + bcc1) - bcc[j];
                }
                if (is_tile) {
                    if (sp >= s_begin && sp < s_end) {
                        st_rows<C>(d_br, o_sp, brr, is_tile, P);
                        st_rows<C>(d_bc, o_sp, bcc, is_tile, P);
                    }
                    const int so = s - 2;
                    if (so >= s_begin && so < s_end) {
                        float dv[C];
#pragma unroll
                        for (int j = 0; j < C; ++j) {
                            dv[j] = dvp[j] + bss_cur[j];
                            dv[j] = dv[j] - bss_old[j];
                        }
                        const unsigned int o = o_sp - plane_stride;
                        if constexpr (EPI == EPI_COLD) {
                            float g_o[C], v_o[C];
#pragma unroll
                            for (int j = 0; j < C; ++j) {
                                const float csv = tv[1][j], ctv = tv[2][j];
                                const float u = cold_u(tv[0][j]), ucc = u * inv_cc;
                                float ps_n = ((cold_pt(tv[0][j], ctv) - ucc) + dv[j]) + inv_cc;
                                ps_n = fminf(ps_n, csv);
                                float pt_n = (ps_n + ucc) - dv[j];
                                pt_n = fminf(pt_n, ctv);
                                const float e = cc * ((pt_n + dv[j]) - ps_n);
                                erru += fabsf(e);
                                float u_n = u - e;
                                v_o[j] = cold_v(pt_n, ctv, u_n);
                                g_o[j] = dv[j] - ((ps_n - pt_n) + u_n * inv_cc);
                            }
                            st_rows<C>(d_s0, o, g_o, is_tile, P);
                            st_rows<C>(d_s1, o, v_o, is_tile, P);
                        } else if constexpr (TWIN) {
                            float g_o[C], pt_o[C], u_o[C];
                            const float one_over_cc = P.inv_cc_l;
#pragma unroll
                            for (int j = 0; j < C; ++j) {
                                const float u = tv[TS_S2][j], uc = div_cc<true>(u, cc, inv_cc);
                                const float ps_n = min_twin(((dv[j] + tv[TS_S1][j]) - uc) + one_over_cc,
                                                            tv[TS_CS][j]);
                                pt_o[j] = min_twin((-dv[j] + ps_n) + uc, tv[TS_CT][j]);
                                const float e = cc * ((dv[j] + pt_o[j]) - ps_n);
                                if (j == 0 || in_r[j])
                                    errp.add(fabsf(e));
                                u_o[j] = u - e;
                                g_o[j] = dv[j] - ((ps_n - pt_o[j]) + div_cc<true>(u_o[j], cc, inv_cc));
                            }
                            st_rows<C>(d_s0, o, g_o, is_tile, P);
                            st_rows<C>(d_s1, o, pt_o, is_tile, P);
                            st_rows<C>(d_s2, o, u_o, is_tile, P);
                        } else if constexpr (EPI == EPI_BINARY) {
                            float g_o[C], pt_o[C], u_o[C];
#pragma unroll
                            for (int j = 0; j < C; ++j) {
                                const float ucc = div_cc<EXACT>(tv[TS_S2][j], cc, inv_cc);
                                float ps_n = ((tv[TS_S1][j] - ucc) + dv[j]) + inv_cc;
                                ps_n = min_sel<EXACT>(ps_n, tv[TS_CS][j]);
                                float pt_n = (ps_n + ucc) - dv[j];
                                pt_n = min_sel<EXACT>(pt_n, tv[TS_CT][j]);
                                const float e = cc * ((pt_n + dv[j]) - ps_n);
                                // cells past the last row hold zero state
                                // and add nothing
                                erru += abs_ref(e);
                                pt_o[j] = pt_n;
                                u_o[j] = tv[TS_S2][j] - e;
                                g_o[j] = dv[j] - ((ps_n - pt_n) + div_cc<EXACT>(u_o[j], cc, inv_cc));
                            }
                            st_rows<C>(d_s0, o, g_o, is_tile, P);
                            st_rows<C>(d_s1, o, pt_o, is_tile, P);
                            st_rows<C>(d_s2, o, u_o, is_tile, P);
                        } else {
                            st_rows<C>(d_s0, o, dv, is_tile, P);
                        }
                    }
                }
#pragma unroll
                for (int j = 0; j < C; ++j)
                    dvp[j] = dn[j];
            }
#pragma unroll
            for (int j = 0; j < C; ++j) {
                br_prev[j] = br[j];
                bc_prev[j] = bc[j];
                bcr_prev[j] = bcr[j];
            }
            brd_prev = brd;
            o_sp += plane_stride;
        }
        __syncthreads();  // stage slots and factor planes are reused by the next item
        if constexpr (TWIN)
            finish_item<NT, true>(errp, P, li, it, B.done_count, s_red, &s_is_last);
        else if constexpr (BIN)
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

}  // namespace asets
