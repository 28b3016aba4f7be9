// small_grid.cuh -- the device time loop of a small grid as one kernel.
//
// A marching tile (step_kernels.cuh) walks down its rows, so a step of a small
// grid takes as long as one tile's march however few tiles there are, and
// every attempt pays two or three kernel launches on top: 9 + 3 us of a
// 200^2 acoustics step of 12 us whose arithmetic is 0.2 us of the chip.  Here
// one cooperative kernel runs the attempts in a loop.  A CTA holds a tile of
// 32 x NY cells, one per thread, with its two halo cells on each side (28 x
// (NY - 4) are written), so all rows of the tile are worked on at once; a warp is
// one row, so the x sweep exchanges within the warp and only the y sweep
// needs the CTA's barriers (three a tile).  Ghost cells are not filled but
// read from the interior cell their boundary rule names.  Between attempts
// the CTAs meet at a barrier in global memory, after which each works out the
// reference's accept/reject and dt for itself from the attempt's Courant
// number (the same numbers in every CTA), so nothing returns to the host
// before the loop is done.
//
// The halo makes a tile compute 32 NY cells to write 28 (NY - 4), so the
// marching kernels win once the grid fills the chip several times over:
// see small_grid_fits (claw2.cu) for where the line lies.
#pragma once

#include "step_kernels.cuh"

namespace claw2 {

// Rotating words of the attempts: attempt k uses entry k % 3, and entry
// (k + 2) % 3 is cleared after the barrier of attempt k (its last readers, of
// attempt k - 1, have arrived by then; its next users start after the next barrier).
struct SmallCtl {
    unsigned int arrived;  // barrier: arrivals so far
    int pad;
    unsigned long long cfl[3];
    int status[3];
};

template <class RP, int NY>
struct SmallSmem {
    static constexpr int NT = 32 * NY;
    double cell[RP::NC][NT];
    double wx[Lim<RP>::N][NT], wy[Lim<RP>::N][NT];  // limiter records of the x and y interfaces
    double up[RP::MEQN][NT], dn[RP::MEQN][NT];      // increments for the row below (row - 1) and the row above
    // the next tile's cells on their way from memory: q, then the aux data (each thread its own)
    double stage[RP::MEQN + AuxTraits<RP>::MAUX][NT];
    double red[NY];
    EvolveDev e;
    int go;
};

// 8 bytes from global to shared memory, asynchronously (waited for by copy_wait)
__device__ __forceinline__ void copy_async(double* dst, const double* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void copy_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// One unsplit step of the tile's cells: v receives the new value of this
// thread's cell (meaningful on the tile's inner cells).
template <class RP, int NY, int SPEC>
__device__ __forceinline__ void small_unsplit(const StepArgs& a, SmallSmem<RP, NY>& S, const double (&c)[RP::NC],
                                              int cp, int r, double dtdx, double dtdy,
                                              double& cfl, double (&v)[RP::MEQN]) {
    constexpr int ME = RP::MEQN, MW = RP::MWAVES, NC = RP::NC, NL = Lim<RP>::N;
    constexpr bool TAUX = AuxTraits<RP>::TRANSVERSE_AUX;
    constexpr bool ZS = SkipTraits<RP>::OK && AuxTraits<RP>::MAUX == 0;
    using Iface = typename RP::Iface;
    const int t = threadIdx.x, tx = t & 31, ty = t >> 5;
    const int tl = tx > 0 ? t - 1 : t, tr = tx < 31 ? t + 1 : t;
    const int tb = ty > 0 ? t - 32 : t, ta = ty < NY - 1 ? t + 32 : t;
    const int mx = a.L.mx, my = a.L.my;
    const RPParams& P = a.rp;
    const int order = (SPEC == SPEC_MC2) ? 2 : a.meth.order;
    const int trans = (SPEC == SPEC_MC2) ? 2 : a.meth.transverse;
    const bool tc = (order > 1) && (trans == 2);
    const bool zs = ZS && (SPEC != SPEC_ANY || a.meth.fwave == 0);
#pragma unroll
    for (int k = 0; k < NC; ++k) S.cell[k][t] = c[k];
    __syncthreads();  // cells of the tile in place

    const double h = 0.5 * dtdx * dtdy;
    double own[ME], ub[ME];  // increments of this cell and of the cell below
    // ---- x: the interface (cp-1 | cp) of the cell's row, solved and finished
    // within the warp (its state is gone before the y work begins) ----
    {
        Iface f;
        double am[ME], ap[ME], n[NC], rec[NL];
#pragma unroll
        for (int k = 0; k < NC; ++k) n[k] = S.cell[k][tl];
        const bool z = ZS && zs && __all_sync(0xffffffffu, same_q<ME, NC>(n, c));
        if (ZS && z) {
            SkipTraits<RP>::template zero_iface<1>(n, c, P, f);
#pragma unroll
            for (int m = 0; m < ME; ++m) am[m] = ap[m] = 0.0;
        } else {
            RP::template solve<1>(n, c, P, f, am, ap);
        }
        // the Courant number over the reference's interface sets (step2.f90:92,172)
        if (tx > 0 && cp >= 2 && cp <= mx + 2 && r >= 1 && r <= my + 2) cfl = fmax(cfl, iface_cfl<RP, 1>(f, P, dtdx));
        double xl[ME], bl[ME], dl[ME], dn[ME];  // left neighbour's row, below-left, above-left, above
#pragma unroll
        for (int m = 0; m < ME; ++m) own[m] = ub[m] = xl[m] = bl[m] = dl[m] = dn[m] = 0.0;
        if (!(ZS && z)) {
            double cq[ME];
            if (order != 1) {
                Lim<RP>::template rec<1>(f, P, rec);
#pragma unroll
                for (int k = 0; k < NL; ++k) S.wx[k][t] = rec[k];
                __syncwarp();
                double s[MW], num[MW];
                RP::template speeds<1>(f, P, s);
                Lim<RP>::up(rec, s, [&](int j, bool left) { return S.wx[j][left ? tl : tr]; }, num);
                correction<RP, 1, SPEC>(f, P, a.meth, dtdx, rec, s, num, cq);
            } else {
#pragma unroll
                for (int m = 0; m < ME; ++m) cq[m] = 0.0;
            }
#pragma unroll
            for (int m = 0; m < ME; ++m) {
                const double g = 0.5 * cq[m];
                own[m] = -dtdx * (ap[m] - g);
                xl[m] = -dtdx * (am[m] + g);
            }
            if (trans > 0) {
                double as2[ME], bm[ME], bp[ME];
#pragma unroll
                for (int m = 0; m < ME; ++m) as2[m] = tc ? am[m] + cq[m] : am[m];
                if constexpr (TAUX) {
                    double cm[NC], cu[NC];
                    const int lb = tx > 0 ? tb - 1 : tb, la = tx > 0 ? ta - 1 : ta;
#pragma unroll
                    for (int k = 0; k < NC; ++k) {
                        cm[k] = S.cell[k][lb];
                        cu[k] = S.cell[k][la];
                    }
                    rpt2h_aux<RP, 1>(as2, cm, n, cu, h, bm, bp);
                } else {
                    Trans<RP>::template split<1>(f, P, h, as2, bm, bp);  // into column cp-1
                }
#pragma unroll
                for (int m = 0; m < ME; ++m) {
                    xl[m] = xl[m] + (bp[m] - bm[m]);
                    bl[m] = bm[m];
                    dl[m] = -bp[m];
                }
#pragma unroll
                for (int m = 0; m < ME; ++m) as2[m] = tc ? ap[m] - cq[m] : ap[m];
                if constexpr (TAUX) {
                    double cm[NC], cu[NC];
#pragma unroll
                    for (int k = 0; k < NC; ++k) {
                        cm[k] = S.cell[k][tb];
                        cu[k] = S.cell[k][ta];
                    }
                    rpt2h_aux<RP, 1>(as2, cm, c, cu, h, bm, bp);
                } else {
                    Trans<RP>::template split<1>(f, P, h, as2, bm, bp);  // into column cp
                }
#pragma unroll
                for (int m = 0; m < ME; ++m) {
                    own[m] = own[m] + (bp[m] - bm[m]);
                    ub[m] = bm[m];
                    dn[m] = -bp[m];
                }
            }
        }
        // the right neighbour's left-going parts
#pragma unroll
        for (int m = 0; m < ME; ++m) {
            own[m] = own[m] + __shfl_down_sync(0xffffffffu, xl[m], 1);
            ub[m] = ub[m] + __shfl_down_sync(0xffffffffu, bl[m], 1);
            S.dn[m][t] = dn[m] + __shfl_down_sync(0xffffffffu, dl[m], 1);
        }
    }
    // ---- y: the interface (r-1 | r) of the cell's column ----
    Iface fY;
    double amY[ME], apY[ME];
    bool zY;
    {
        double n[NC], cc[NC];
#pragma unroll
        for (int k = 0; k < NC; ++k) {
            n[k] = S.cell[k][tb];
            cc[k] = S.cell[k][t];
        }
        zY = ZS && zs && __all_sync(0xffffffffu, same_q<ME, NC>(n, cc));
        if (ZS && zY) {
            SkipTraits<RP>::template zero_iface<2>(n, cc, P, fY);
#pragma unroll
            for (int m = 0; m < ME; ++m) amY[m] = apY[m] = 0.0;
        } else {
            RP::template solve<2>(n, cc, P, fY, amY, apY);
        }
        double rec[NL];
        Lim<RP>::template rec<2>(fY, P, rec);
#pragma unroll
        for (int k = 0; k < NL; ++k) S.wy[k][t] = rec[k];
    }
    if (ty > 0 && r >= 2 && r <= my + 2 && cp >= 1 && cp <= mx + 2) cfl = fmax(cfl, iface_cfl<RP, 2>(fY, P, dtdy));
    __syncthreads();  // limiter records in place
    double yl[ME], yr[ME], bl2[ME], br2[ME];  // y: left and right neighbour on this row, and on the row below
#pragma unroll
    for (int m = 0; m < ME; ++m) yl[m] = yr[m] = bl2[m] = br2[m] = 0.0;
    if (!(ZS && zY)) {
        double cq[ME];
        if (order != 1) {
            double rec[NL], s[MW], num[MW];
            Lim<RP>::template rec<2>(fY, P, rec);
            RP::template speeds<2>(fY, P, s);
            Lim<RP>::up(rec, s, [&](int j, bool left) { return S.wy[j][left ? tb : ta]; }, num);
            correction<RP, 2, SPEC>(fY, P, a.meth, dtdy, rec, s, num, cq);
        } else {
#pragma unroll
            for (int m = 0; m < ME; ++m) cq[m] = 0.0;
        }
#pragma unroll
        for (int m = 0; m < ME; ++m) {
            const double f = 0.5 * cq[m];
            own[m] = own[m] - dtdy * (apY[m] - f);
            ub[m] = ub[m] - dtdy * (amY[m] + f);
        }
        if (trans > 0) {
            double as2[ME], bm[ME], bp[ME];
#pragma unroll
            for (int m = 0; m < ME; ++m) as2[m] = tc ? amY[m] + cq[m] : amY[m];
            if constexpr (TAUX) {
                double cm[NC], c0[NC], cu[NC];
                const int bl1 = tx > 0 ? tb - 1 : tb, br1 = tx < 31 ? tb + 1 : tb;
#pragma unroll
                for (int k = 0; k < NC; ++k) {
                    cm[k] = S.cell[k][bl1];
                    c0[k] = S.cell[k][tb];
                    cu[k] = S.cell[k][br1];
                }
                rpt2h_aux<RP, 2>(as2, cm, c0, cu, h, bm, bp);
            } else {
                Trans<RP>::template split<2>(fY, P, h, as2, bm, bp);  // into row r-1
            }
#pragma unroll
            for (int m = 0; m < ME; ++m) {
                ub[m] = ub[m] + (bp[m] - bm[m]);
                bl2[m] = bm[m];
                br2[m] = -bp[m];
            }
#pragma unroll
            for (int m = 0; m < ME; ++m) as2[m] = tc ? apY[m] - cq[m] : apY[m];
            if constexpr (TAUX) {
                double cm[NC], cu[NC];
#pragma unroll
                for (int k = 0; k < NC; ++k) {
                    cm[k] = S.cell[k][tl];
                    cu[k] = S.cell[k][tr];
                }
                double c0[NC];
#pragma unroll
                for (int k = 0; k < NC; ++k) c0[k] = S.cell[k][t];
                rpt2h_aux<RP, 2>(as2, cm, c0, cu, h, bm, bp);
            } else {
                Trans<RP>::template split<2>(fY, P, h, as2, bm, bp);  // into row r
            }
#pragma unroll
            for (int m = 0; m < ME; ++m) {
                own[m] = own[m] + (bp[m] - bm[m]);
                yl[m] = bm[m];
                yr[m] = -bp[m];
            }
        }
    }
#pragma unroll
    for (int m = 0; m < ME; ++m) {
        own[m] = own[m] + __shfl_down_sync(0xffffffffu, yl[m], 1) + __shfl_up_sync(0xffffffffu, yr[m], 1);
        ub[m] = ub[m] + __shfl_down_sync(0xffffffffu, bl2[m], 1) + __shfl_up_sync(0xffffffffu, br2[m], 1);
        S.up[m][t] = ub[m];
    }
    __syncthreads();  // increments for the rows above and below in place
#pragma unroll
    for (int m = 0; m < ME; ++m) v[m] = S.cell[m][t] + ((own[m] + S.up[m][ta]) + S.dn[m][tb]);
}

// One split step (x sweep, then y sweep) of the tile's cells.
template <class RP, int NY, int SPEC>
__device__ __forceinline__ void small_split(const StepArgs& a, SmallSmem<RP, NY>& S, const double (&q)[RP::MEQN],
                                            const double (&c)[RP::NC], const double (&av)[AuxTraits<RP>::MAUX > 0
                                                                                              ? AuxTraits<RP>::MAUX
                                                                                              : 1],
                                            int cp, int r, double dtdx, double dtdy, double& cfl,
                                            double (&v)[RP::MEQN]) {
    constexpr int ME = RP::MEQN, MW = RP::MWAVES, NC = RP::NC, NL = Lim<RP>::N;
    constexpr bool ZS = SkipTraits<RP>::OK && AuxTraits<RP>::MAUX == 0;
    using Iface = typename RP::Iface;
    const int t = threadIdx.x, tx = t & 31, ty = t >> 5;
    const int tl = tx > 0 ? t - 1 : t, tr = tx < 31 ? t + 1 : t;
    const int tb = ty > 0 ? t - 32 : t, ta = ty < NY - 1 ? t + 32 : t;
    const int mx = a.L.mx, my = a.L.my;
    const RPParams& P = a.rp;
    const bool zs = ZS && (SPEC != SPEC_ANY || a.meth.fwave == 0);
    const bool second = (SPEC != SPEC_ANY) || a.meth.order != 1;
    // x: a warp is a row, so nothing leaves it
    double q1[ME];
    {
        Iface f;
        double am[ME], ap[ME], n[NC], cq[ME], rec[NL];
#pragma unroll
        for (int k = 0; k < NC; ++k) n[k] = __shfl_up_sync(0xffffffffu, c[k], 1);
        const bool z = ZS && zs && __all_sync(0xffffffffu, tx == 0 || same_q<ME, NC>(n, c));
        if (ZS && z) {
            SkipTraits<RP>::template zero_iface<1>(n, c, P, f);
#pragma unroll
            for (int m = 0; m < ME; ++m) am[m] = ap[m] = 0.0;
        } else {
            RP::template solve<1>(n, c, P, f, am, ap);
        }
        if (tx > 0 && cp >= 2 && cp <= mx + 2) cfl = fmax(cfl, iface_cfl<RP, 1>(f, P, dtdx));
#pragma unroll
        for (int m = 0; m < ME; ++m) cq[m] = 0.0;
        if (second && !(ZS && z)) {
            Lim<RP>::template rec<1>(f, P, rec);
#pragma unroll
            for (int k = 0; k < NL; ++k) S.wx[k][t] = rec[k];
            __syncwarp();
            double s[MW], num[MW];
            RP::template speeds<1>(f, P, s);
            Lim<RP>::up(rec, s, [&](int j, bool left) { return S.wx[j][left ? tl : tr]; }, num);
            correction<RP, 1, SPEC>(f, P, a.meth, dtdx, rec, s, num, cq);
        }
        const bool inner = cp >= 2 && cp <= mx + 1;  // ghost columns keep their values
#pragma unroll
        for (int m = 0; m < ME; ++m) {
            const double left = __shfl_down_sync(0xffffffffu, -dtdx * (am[m] + 0.5 * cq[m]), 1);
            q1[m] = inner ? q[m] + (-dtdx * (ap[m] - 0.5 * cq[m]) + left) : q[m];
        }
    }
    // y, from the x-swept cells
    double c1[NC];
    AuxTraits<RP>::prep(q1, av, P, c1);
#pragma unroll
    for (int k = 0; k < NC; ++k) S.cell[k][t] = c1[k];
    __syncthreads();  // x-swept cells in place
    Iface f;
    double am[ME], ap[ME];
    bool z;
    {
        double n[NC], rec[NL];
#pragma unroll
        for (int k = 0; k < NC; ++k) n[k] = S.cell[k][tb];
        z = ZS && zs && __all_sync(0xffffffffu, same_q<ME, NC>(n, c1));
        if (ZS && z) {
            SkipTraits<RP>::template zero_iface<2>(n, c1, P, f);
#pragma unroll
            for (int m = 0; m < ME; ++m) am[m] = ap[m] = 0.0;
        } else {
            RP::template solve<2>(n, c1, P, f, am, ap);
        }
        Lim<RP>::template rec<2>(f, P, rec);
#pragma unroll
        for (int k = 0; k < NL; ++k) S.wy[k][t] = rec[k];
    }
    // (halo columns of the tile have no complete x sweep; the grid's own ghost columns are unchanged by it)
    const bool swept = (tx >= 2 && tx <= 29) || cp < 2 || (cp >= mx + 2 && cp <= mx + 3);
    if (ty > 0 && swept && r >= 2 && r <= my + 2 && cp <= mx + 3) cfl = fmax(cfl, iface_cfl<RP, 2>(f, P, dtdy));
    __syncthreads();  // limiter records in place
    double cq[ME];
#pragma unroll
    for (int m = 0; m < ME; ++m) cq[m] = 0.0;
    if (second && !(ZS && z)) {
        double rec[NL], s[MW], num[MW];
        Lim<RP>::template rec<2>(f, P, rec);
        RP::template speeds<2>(f, P, s);
        Lim<RP>::up(rec, s, [&](int j, bool left) { return S.wy[j][left ? tb : ta]; }, num);
        correction<RP, 2, SPEC>(f, P, a.meth, dtdy, rec, s, num, cq);
    }
#pragma unroll
    for (int m = 0; m < ME; ++m) S.up[m][t] = -dtdy * (am[m] + 0.5 * cq[m]);
    __syncthreads();  // increments for the row below in place
#pragma unroll
    for (int m = 0; m < ME; ++m) v[m] = q1[m] + (-dtdy * (ap[m] - 0.5 * cq[m]) + S.up[m][ta]);
}

// The loop.  Cooperative launch (every CTA resident); `rec` holds the loop's
// record, read at the start and written at the end; `ctl` is zero on entry.
// At most `budget` attempts; a barrier that gives up sets fault bit 1
// (CLAW2_ETIMEOUT) and ends the loop.
template <class RP, int NY, int SPEC, bool SPLIT>
__global__ void __launch_bounds__(32 * NY, 1) k_small_evolve(const StepArgs a, const BCArgs bc, EvolveDev* rec,
                                                             SmallCtl* ctl, int budget) {
    constexpr int ME = RP::MEQN, NC = RP::NC;
    constexpr int MAD = AuxTraits<RP>::MAUX > 0 ? AuxTraits<RP>::MAUX : 1;
    constexpr int TX = 28, TY = NY - 4;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    SmallSmem<RP, NY>& S = *reinterpret_cast<SmallSmem<RP, NY>*>(smem_raw);
    const int t = threadIdx.x, tx = t & 31, ty = t >> 5;
    const int mx = a.L.mx, my = a.L.my, pitch = a.L.pitch;
    const long long plane = a.L.plane;
    const int ntx = (mx + TX - 1) / TX, ntiles = ntx * ((my + TY - 1) / TY);
    if (t == 0) S.e = *rec;
    __syncthreads();
    for (int k = 0; k < budget; ++k) {
        if (S.e.done) break;  // (the same in every CTA)
        const double dtdx = S.e.dtdx, dtdy = S.e.dtdy;
        const double* qo = S.e.cur ? a.qold2 : a.qold;
        double* qn = S.e.cur ? a.qnew2 : a.qnew;
        double cfl = 0.0;
        bool bad = false;
        // Each thread's cell of the next tile is on its way while this tile is
        // worked on (the loads' latency was a tenth of a tile).
        auto fetch = [&](int tile) {
            const int cp = min((tile % ntx) * TX + tx, mx + 3), r = min((tile / ntx) * TY + ty, my + 3);
            bool fx, fy;
            const int cs = bc_src(cp, mx, bc.bcl[0], bc.bcu[0], fx);
            const int rs = bc_src(r, my, bc.bcl[1], bc.bcu[1], fy);
            const double* src = qo + (long long)rs * pitch + cs;
#pragma unroll
            for (int m = 0; m < ME; ++m) copy_async(&S.stage[m][t], src + m * plane);
            if constexpr (AuxTraits<RP>::MAUX > 0) {
                const double* ax = a.aux + (long long)r * pitch + cp;
#pragma unroll
                for (int m = 0; m < MAD; ++m) copy_async(&S.stage[ME + m][t], ax + m * plane);
            }
        };
        if ((int)blockIdx.x < ntiles) fetch(blockIdx.x);
        for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
            const int cp0 = (tile % ntx) * TX + tx, r0 = (tile / ntx) * TY + ty;  // padded position
            const int cp = min(cp0, mx + 3), r = min(r0, my + 3);
            bool fx, fy;  // a wall mirrored this cell
            bc_src(cp, mx, bc.bcl[0], bc.bcu[0], fx);
            bc_src(r, my, bc.bcl[1], bc.bcu[1], fy);
            double q[ME], c[NC], av[MAD], v[ME];
            copy_wait();
#pragma unroll
            for (int m = 0; m < ME; ++m) {
                double x = S.stage[m][t];
                if (fx && m == 1) x = -x;
                if (fy && m == 2) x = -x;
                q[m] = x;
            }
#pragma unroll
            for (int m = 0; m < MAD; ++m) av[m] = AuxTraits<RP>::MAUX > 0 ? S.stage[ME + m][t] : 0.0;
            if (tile + (int)gridDim.x < ntiles) fetch(tile + gridDim.x);
            AuxTraits<RP>::prep(q, av, a.rp, c);
            // (positions past the grid, cp0 > mx + 3 or r0 > my + 3, work on copies of the last ghost cell and
            // count for nothing)
            if constexpr (SPLIT) small_split<RP, NY, SPEC>(a, S, q, c, av, cp0, r0, dtdx, dtdy, cfl, v);
            else small_unsplit<RP, NY, SPEC>(a, S, c, cp0, r0, dtdx, dtdy, cfl, v);
            if (tx >= 2 && tx < 30 && ty >= 2 && ty < NY - 2 && cp0 <= mx + 1 && r0 <= my + 1) {
                double* dst = qn + (long long)r0 * pitch + cp0;
#pragma unroll
                for (int m = 0; m < ME; ++m) dst[m * plane] = v[m];
                bad = bad || !all_finite<ME>(v);
            }
        }
        const int w = k % 3;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) cfl = fmax(cfl, __shfl_xor_sync(0xffffffffu, cfl, o));
        if (tx == 0) S.red[ty] = cfl;
        if (__any_sync(0xffffffffu, bad) && tx == 0) atomicOr(&ctl->status[w], 1);
        __syncthreads();
        if (t == 0) {
            double m = 0.0;
            for (int i = 0; i < NY; ++i) m = fmax(m, S.red[i]);
            atomicMax(&ctl->cfl[w], (unsigned long long)__double_as_longlong(m));
            // the barrier: arrive, then wait until every CTA has
            __threadfence();
            atomicAdd(&ctl->arrived, 1u);
            const unsigned int target = (unsigned int)(k + 1) * gridDim.x;
            int spins = 0;
            while (ld_acquire(&ctl->arrived) < target && ++spins < GRID_SPIN_LIMIT) {}
            EvolveDev& e = S.e;
            if (spins >= GRID_SPIN_LIMIT) {
                e.fault = 2;
                e.done = 1;
            } else {
                const double got = __longlong_as_double((long long)__ldcg(&ctl->cfl[w]));
                const int st = __ldcg(&ctl->status[w]);
                evolve_finish(e, got, st);
                if (blockIdx.x == 0) {  // (see SmallCtl)
                    const int z = (k + 2) % 3;
                    ctl->cfl[z] = 0ull;
                    ctl->status[z] = 0;
                }
            }
        }
        __syncthreads();
    }
    if (blockIdx.x == 0 && t == 0) *rec = S.e;
}

}  // namespace claw2
