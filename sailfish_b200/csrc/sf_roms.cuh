// ROMS-form barotropic step (the "roms" semantics): the free-surface / depth-integrated
// momentum step of ROMS's step2d_LF_AM3, which the reference carries only as untranslated
// Fortran (obsolete/step2d_LF_AM3.h.py), with its 2D Coriolis (:1503-1530), surface stress
// (:2598-2612), quadratic bottom drag (nonlinear/set_vbc.py:16-41) and the fast-time averages
// Zt_avg1, DU_avg1/2, DV_avg1/2 (:778-846), for closed rectangular basins.  It exists beside
// the reference-semantics kernels because the benchmark configurations need forcing, Coriolis
// and a stable step, none of which the reference's runnable 2D kernels have.
//
// Divisions go through ddiv: IEEE in FP64, the fast FP32 division (__fdividef) in FP32.
//
// Index conventions as the rest of the package: flat p = j*I + i over (M+1) x (L+1) rho points;
// ubar(p) on the west face of rho p, vbar(p) on its south face; interior rho i = 1..I-2,
// j = 1..J-2; interior U faces i = 2..I-2 (walls i = 1, I-1), V faces j = 2..J-2.
//
// A substep has a predictor and a corrector, each the free surface, then the momentum.  Its forms, of the
// same bits: in one launch on tiles (roms_sub_tile); in two, a phase each, by warps that walk up the rows
// of a strip of columns (roms_phase_rows); in four, a point a thread (roms_zeta_point, roms_mom_point).
// Time levels: slots b (n-1), n and p (the predicted n+1*); the phases' corrector writes n+1 into b and
// the host swaps b and n (the tiles' levels: roms_sub_tile).  Every expression keeps the operand
// order of the oracle's restatement (oracle/roms_oracle.py), so the FP64 build (no FMA contraction)
// reproduces it bit for bit; the fast-time averages are FP64 in both precisions.
#pragma once

namespace sf {


// The barotropic substep's products and sums, with the FP32 form's contractions written out: a product
// either rounds by itself (rmul) or goes into one fused multiply-add (rfma), so that every form of
// the substep (two launches, fused; single grid, ensemble) gives the same bits whatever the compiler
// would fuse in it.  The FP64 form rounds every product and sum, as the oracle does.
template <typename R>
__device__ __forceinline__ R rmul(R a, R b) {
    if constexpr (sizeof(R) == 4) return __fmul_rn(a, b);
    else return a * b;
}
template <typename R>
__device__ __forceinline__ R rfma(R a, R b, R c) {
    if constexpr (sizeof(R) == 4) return __fmaf_rn(a, b, c);
    else return a * b + c;
}
// an FP64 average plus a weighted term
template <typename R>
__device__ __forceinline__ double rsum(double s, double c, double x) {
    if constexpr (sizeof(R) == 4) return __fma_rn(c, x, s);
    else return s + c * x;
}
template <typename R>
__device__ __forceinline__ R roms_am3(R r, R rn, R rb) {
    return rfma(-R(1.0 / 12.0), rb, rfma(R(5.0 / 12.0), r, rmul(R(8.0 / 12.0), rn)));
}
// The momentum right-hand side at a face: gm, hm the pressure-gradient surface and depth on its minus
// side, gp, h on its plus side; u the velocity there, o4 the four-point average of the other
// component; cor the sum of the two Coriolis fluxes; area 4 / ((pm + pm)(pn + pn)).
template <typename R, bool V>
__device__ __forceinline__ R roms_rhs(R met, R gm, R gp, R hm, R h, R cor, R u, R o4, R rdrag2, R str, R area) {
    const R cffg = R(0.5 * 10.0);   // 0.5 g, g = 10 (mod_constants.py:26)
    const R in = rfma(hm + h, gm - gp, rfma(gm, gm, -rmul(gp, gp)));
    const R pa = rmul(cffg, met);
    const R pc = V ? rmul(pa, in) + rmul(R(-0.5), cor) : rfma(pa, in, rmul(R(0.5), cor));
    const R tau = rfma(-rmul(rdrag2, u), sqrt(rfma(u, u, rmul(o4, o4))), str);
    return rfma(tau, area, pc);
}
// A face's new velocity: (u Ds + pmn2 cdt f) / Dn.
template <typename R>
__device__ __forceinline__ R roms_new(R u, R Ds, R pmn2, R cdt, R f, R Dn) {
    return ddiv(rfma(rmul(pmn2, cdt), f, rmul(u, Ds)), Dn);
}

// One phase of a substep on a strip of columns.  A warp owns the 29 columns i0 .. i0 + 28 (lane l is
// column i0 + l - 2; lanes 0, 1 and 31 hold the neighbours) and walks up `nrows` rows from j0,
// starting one row below for the free surface that the first row's V faces need.  West and east
// neighbours come from the next lanes by shuffle, the southern ones from the row before, so a node's
// inputs are loaded once (plus 3 columns in 32 and one row in nrows + 1), with no shared memory and no
// barrier, and the new free surface is used by the momentum step from registers.
//
// The corrector also adds the fast-time averages, the predictor's terms (fields of level n, which
// the substep does not change) and its own, in that order: one read and one write of the five FP64
// averages per substep.  Neither phase reads a slot it writes (the predictor writes p and the
// tendencies of level n, the corrector b), so warps are independent.
//
// Ring nodes of the free surface take the value of the nearest interior node (zero gradient at the
// closed walls): its owner writes them.
// Bound: bytes per node and substep 252 in FP32 (80 predictor, 172 corrector of which 80 the
// averages), 424 in FP64.
template <typename R>
struct RomsRow {   // a node's inputs of one row
    R z, h, v, om;                       // row j + 1: flux level's zeta and vbar, depth, om_v
    R u, on, pm, pn, zk;                 // row j: flux level's ubar, metrics, zeta(kstp)
    R fo, uk, vk, su, sv;                // row j, momentum only
    R zrn, zrb, run, rub, rvn, rvb;      // corrector: tendencies of levels n and n-1
};

template <typename R, int PH>
__device__ __forceinline__ void roms_load(const Geo<R> &g, const RomsArgs<R> &a, int il, int j, bool mom,
                                          RomsRow<R> &w) {
    const int J = g.J;
    const int jc = j < 0 ? 0 : (j > J - 1 ? J - 1 : j);
    const int jn = j + 1 < 0 ? 0 : (j + 1 > J - 1 ? J - 1 : j + 1);
    const int p = jc * g.I + il, n = jn * g.I + il;
    w.z = a.zrhs[n];
    w.v = a.vrhs[n];
    w.h = g.h[n];
    w.om = g.om_v[n];
    w.u = a.urhs[p];
    w.on = g.on_u[p];
    w.pm = g.pm[p];
    w.pn = g.pn[p];
    w.zk = a.zkstp[p];
    w.fo = g.fomn[p];
    if (PH == 1 && !a.first) {
        w.zrn = a.rz_n[p];
        w.zrb = a.rz_b[p];
    }
    if (mom) {
        w.uk = a.ukstp[p];
        w.vk = a.vkstp[p];
        w.su = a.sustr[p];
        w.sv = a.svstr[p];
        if (PH == 1 && !a.first) {
            w.run = a.ru_n[p];
            w.rub = a.ru_b[p];
            w.rvn = a.rv_n[p];
            w.rvb = a.rv_b[p];
        }
    }
}

template <typename R, int PH>
__device__ __forceinline__ void roms_phase_rows(const Geo<R> &g, const RomsArgs<R> &a, const int i0,
                                                const int j0, const int nrows) {
    const int I = g.I, J = g.J, lane = threadIdx.x & 31;
    if (j0 >= J) return;   // whole warp
    const int i = i0 - 2 + lane, il = i < 0 ? 0 : (i > I - 1 ? I - 1 : i);
    const bool out = lane >= 2 && lane <= 30 && i < I;
    const int jend = j0 + nrows < J ? j0 + nrows : J;
    auto west = [](R x) { return __shfl_up_sync(0xffffffffu, x, 1); };
    auto east = [](R x) { return __shfl_down_sync(0xffffffffu, x, 1); };
    const R rdrag2 = (R)a.rdrag2, dt = (R)a.dtfast;
    const R dtz = PH == 0 && !a.first ? (R)(2.0 * a.dtfast) : dt;
    const R cdt = PH == 0 && !a.first ? dt : (R)(0.5 * a.dtfast);
    RomsRow<R> w;
    // the row below the first: its southern values come from the load of the row before it
    roms_load<R, PH>(g, a, il, j0 - 2, false, w);
    R zc = w.z, hc = w.h, vc = w.v, omc = w.om;
    R dvc, zks;   // DVom at row j; zeta(kstp) + h one row south
    {
        const int js = j0 - 2 < 0 ? 0 : j0 - 2;
        const R Ds = a.zrhs[js * I + il] + g.h[js * I + il];
        dvc = rmul(rmul(vc, rmul(R(0.5), (zc + hc) + Ds)), omc);
        zks = R(0);
    }
    R gs = R(0), hs = R(0), dzs = R(0), vfs = R(0), us = R(0), ues = R(0), pms = R(1), pns = R(1);
    roms_load<R, PH>(g, a, il, j0 - 1, false, w);
    for (int j = j0 - 1; j < jend; ++j) {
        const RomsRow<R> c = w;
        if (j + 1 < jend) roms_load<R, PH>(g, a, il, j + 1, true, w);   // the next row's, in flight
        const bool mine = out && j >= j0;
        const int p = j * I + i;
        double A[5];
        if (PH == 1 && a.acc == 1 && mine) {
            A[0] = a.Zt[p];
            A[1] = a.DU1[p];
            A[2] = a.DV1[p];
            A[3] = a.DU2[p];
            A[4] = a.DV2[p];
        }
        // free surface
        const R Dc = zc + hc, Dw = west(Dc);
        const R au = rmul(c.u, rmul(R(0.5), Dc + Dw)), du = rmul(au, c.on);
        const R dvn = rmul(rmul(c.v, rmul(R(0.5), (c.z + c.h) + Dc)), c.om);
        const R rz = rfma(-east(au), east(c.on), du) + (dvc - dvn);
        R f = rz;
        if (PH == 1 && !a.first) f = roms_am3(rz, c.zrn, c.zrb);
        const R znew = rfma(rmul(rmul(c.pm, c.pn), dtz), f, c.zk);
        // the pressure-gradient surface
        R gp;
        if (a.first) gp = rmul(R(0.5), c.zk + znew);
        else if (PH == 0) gp = rfma(R(0.68), zc, rmul(R(0.16), c.zk + znew));
        else gp = rfma(R(0.6), znew, rmul(R(0.4), zc));
        const R dk = c.zk + hc, dz = znew + hc;
        const R ue = east(c.u);
        const R fa = rmul(rmul(R(0.5), Dc), c.fo), vf = rmul(fa, c.u + ue);
        if (j >= j0) {   // the whole warp
            const bool ri = i >= 1 && i <= I - 2, rj = j >= 1 && j <= J - 2;
            // U face
            R unew = R(0), runew = R(0);
            {
                const R gw = west(gp), hw = west(hc);
                const R cor = rfma(fa, vc + c.v, west(rmul(fa, vc + c.v)));
                const R pmn2 = rmul(c.pm + west(c.pm), c.pn + west(c.pn));
                const R v4 = rmul(R(0.25), ((vc + c.v) + west(vc)) + west(c.v));
                const R Ds = dk + west(dk), Dn = dz + west(dz);
                if (i >= 2 && ri && rj) {
                    const R ru = roms_rhs<R, false>(c.on, gw, gp, hw, hc, cor, c.u, v4, rdrag2, c.su,
                                                    ddiv(R(4.0), pmn2));
                    R fu = ru;
                    if (PH == 0) runew = ru;
                    else if (!a.first) fu = roms_am3(ru, c.run, c.rub);
                    unew = roms_new(c.uk, Ds, pmn2, cdt, fu, Dn);
                }
            }
            // V face
            R vnew = R(0), rvnew = R(0);
            if (j >= 2 && rj && ri) {
                const R pmn2 = rmul(c.pm + pms, c.pn + pns);
                const R u4 = rmul(R(0.25), ((c.u + ue) + us) + ues);
                const R rv = roms_rhs<R, true>(omc, gs, gp, hs, hc, rfma(fa, c.u + ue, vfs), vc, u4, rdrag2,
                                               c.sv, ddiv(R(4.0), pmn2));
                R fv = rv;
                if (PH == 0) rvnew = rv;
                else if (!a.first) fv = roms_am3(rv, c.rvn, c.rvb);
                vnew = roms_new(c.vk, dk + zks, pmn2, cdt, fv, dz + dzs);
            }
            R dun = R(0), dvnn = R(0);
            if (PH == 1 && a.acc) {   // DUon, DVom of level n (kstp): the predictor's terms
                const R dkw = west(dk);
                dun = i < 1 ? R(0) : rmul(rmul(c.uk, rmul(R(0.5), dk + dkw)), c.on);
                dvnn = j < 1 ? R(0) : rmul(rmul(c.vk, rmul(R(0.5), dk + zks)), omc);
            }
            if (mine) {
                a.uout[p] = unew;
                a.vout[p] = vnew;
                if (PH == 0) {
                    a.ru_n[p] = runew;
                    a.rv_n[p] = rvnew;
                    a.rz_n[p] = ri && rj ? rz : R(0);
                }
                if (ri && rj) {
                    const int di = i == 1 ? -1 : (i == I - 2 ? 1 : 0), dj = j == 1 ? -I : (j == J - 2 ? I : 0);
                    a.zout[p] = znew;
                    if (di) a.zout[p + di] = znew;
                    if (dj) a.zout[p + dj] = znew;
                    if (di && dj) a.zout[p + di + dj] = znew;
                }
                if (PH == 1 && a.acc) {
                    const double dun_ = (double)dun, dvn_ = (double)dvnn;
                    const double dup = i < 1 ? 0.0 : (double)du, dvp = j < 1 ? 0.0 : (double)dvc;
                    if (a.acc == 2) {
                        A[0] = 0.0;
                        A[1] = 0.0;
                        A[2] = 0.0;
                        A[3] = __dmul_rn(a.c2, dun_);
                        A[4] = __dmul_rn(a.c2, dvn_);
                    } else {
                        A[0] = rsum<R>(A[0], a.c1, (double)c.zk);
                        A[1] = rsum<R>(A[1], a.c1, dun_);
                        A[2] = rsum<R>(A[2], a.c1, dvn_);
                        A[3] = rsum<R>(A[3], a.c2, dun_);
                        A[4] = rsum<R>(A[4], a.c2, dvn_);
                    }
                    a.Zt[p] = A[0];
                    a.DU1[p] = A[1];
                    a.DV1[p] = A[2];
                    a.DU2[p] = rsum<R>(A[3], a.c2c, dup);
                    a.DV2[p] = rsum<R>(A[4], a.c2c, dvp);
                }
            }
        }
        // this row becomes the southern one
        gs = gp;
        hs = hc;
        zks = dk;
        dzs = dz;
        vfs = vf;
        us = c.u;
        ues = ue;
        pms = c.pm;
        pns = c.pn;
        dvc = dvn;
        zc = c.z;
        hc = c.h;
        vc = c.v;
        omc = c.om;
    }
}

// One phase of a substep, a point a thread, in two launches: the free surface (with the averages), then the
// momentum, which reads the new free surface.  Every thread loads its neighbours' values and forms their
// fluxes again, but no lane is without a node: strips and tiles hold 29 and 27 columns in 32 lanes, and a basin
// of a few columns (or a few past a strip) leaves most of them idle.  Where it is the faster one:
// roms_by_strips, roms_by_tiles.
//
// The five averages of a node, A as read (acc 1), with the substep's terms: the predictor's (level n: zeta zk,
// face transports dun, dvn), then the corrector's (dup, dvp).
template <typename R>
__device__ __forceinline__ void roms_averages(const RomsArgs<R> &a, const int p, const double *A, const R zk,
                                              const double dun, const double dvn, const double dup, const double dvp) {
    double B[5];
    if (a.acc == 2) {
        B[0] = 0.0;
        B[1] = 0.0;
        B[2] = 0.0;
        B[3] = __dmul_rn(a.c2, dun);
        B[4] = __dmul_rn(a.c2, dvn);
    } else {
        B[0] = rsum<R>(A[0], a.c1, (double)zk);
        B[1] = rsum<R>(A[1], a.c1, dun);
        B[2] = rsum<R>(A[2], a.c1, dvn);
        B[3] = rsum<R>(A[3], a.c2, dun);
        B[4] = rsum<R>(A[4], a.c2, dvn);
    }
    a.Zt[p] = B[0];
    a.DU1[p] = B[1];
    a.DV1[p] = B[2];
    a.DU2[p] = rsum<R>(B[3], a.c2c, dup);
    a.DV2[p] = rsum<R>(B[4], a.c2c, dvp);
}

// The new free surface of interior node p (i, j), also into the ring nodes next to it.
template <typename R>
__device__ __forceinline__ void roms_zeta_out(const Geo<R> &g, R *zout, const int p, const int i, const int j, const R z) {
    const int I = g.I, J = g.J;
    const int di = i == 1 ? -1 : (i == I - 2 ? 1 : 0), dj = j == 1 ? -I : (j == J - 2 ? I : 0);
    zout[p] = z;
    if (di) zout[p + di] = z;
    if (dj) zout[p + dj] = z;
    if (di && dj) zout[p + di + dj] = z;
}

template <typename R>
__device__ __forceinline__ R roms_ubar_D(const Geo<R> &g, const R *z, const R *u, const int p) {   // per on_u
    return rmul(u[p], rmul(R(0.5), (z[p] + g.h[p]) + (z[p - 1] + g.h[p - 1])));
}
template <typename R>
__device__ __forceinline__ R roms_dvom(const Geo<R> &g, const R *z, const R *v, const int p) {
    return rmul(rmul(v[p], rmul(R(0.5), (z[p] + g.h[p]) + (z[p - g.I] + g.h[p - g.I]))), g.om_v[p]);
}
template <typename R, int PH>
__device__ __forceinline__ void roms_zeta_point(const Geo<R> &g, const RomsArgs<R> &a, const long pl) {
    if (pl >= g.s2) return;
    const int p = (int)pl, j = fdiv(p, g.dI), i = p - j * g.I;
    const bool in = i >= 1 && i <= g.I - 2 && j >= 1 && j <= g.J - 2;
    const R du = i < 1 ? R(0) : rmul(roms_ubar_D(g, a.zrhs, a.urhs, p), g.on_u[p]);
    const R dv = j < 1 ? R(0) : roms_dvom(g, a.zrhs, a.vrhs, p);
    if (in) {
        const R rz = rfma(-roms_ubar_D(g, a.zrhs, a.urhs, p + 1), g.on_u[p + 1], du) +
                     (dv - roms_dvom(g, a.zrhs, a.vrhs, p + g.I));
        R f = rz;
        if (PH == 0) a.rz_n[p] = rz;
        else if (!a.first) f = roms_am3(rz, a.rz_n[p], a.rz_b[p]);
        const R dtz = PH == 0 && !a.first ? (R)(2.0 * a.dtfast) : (R)a.dtfast;
        roms_zeta_out(g, a.zout, p, i, j, rfma(rmul(rmul(g.pm[p], g.pn[p]), dtz), f, a.zkstp[p]));
    } else if (PH == 0) {
        a.rz_n[p] = R(0);
    }
    if (PH == 1 && a.acc) {   // level n is the corrector's old level
        double A[5] = {};
        if (a.acc == 1) {
            A[0] = a.Zt[p];
            A[1] = a.DU1[p];
            A[2] = a.DV1[p];
            A[3] = a.DU2[p];
            A[4] = a.DV2[p];
        }
        const R dun = i < 1 ? R(0) : rmul(roms_ubar_D(g, a.zkstp, a.ukstp, p), g.on_u[p]);
        const R dvn = j < 1 ? R(0) : roms_dvom(g, a.zkstp, a.vkstp, p);
        roms_averages(a, p, A, a.zkstp[p], (double)dun, (double)dvn, (double)du, (double)dv);
    }
}
// The pressure-gradient surface of a phase at node q, znew its new free surface.
template <typename R, int PH>
__device__ __forceinline__ R roms_gp(const RomsArgs<R> &a, const int q, const R znew) {
    if (a.first) return rmul(R(0.5), a.zkstp[q] + znew);
    if (PH == 0) return rfma(R(0.68), a.zrhs[q], rmul(R(0.16), a.zkstp[q] + znew));
    return rfma(R(0.6), znew, rmul(R(0.4), a.zrhs[q]));
}
template <typename R, int PH>
__device__ __forceinline__ void roms_mom_point(const Geo<R> &g, const RomsArgs<R> &a, const long pl) {
    if (pl >= g.s2) return;
    const int p = (int)pl, I = g.I, j = fdiv(p, g.dI), i = p - j * I;
    const bool ri = i >= 1 && i <= I - 2, rj = j >= 1 && j <= g.J - 2;
    const R *h = g.h, *u = a.urhs, *v = a.vrhs;
    const R rdrag2 = (R)a.rdrag2, cdt = PH == 0 && !a.first ? (R)a.dtfast : (R)(0.5 * a.dtfast);
    R unew = R(0), runew = R(0), vnew = R(0), rvnew = R(0);
    if (ri && rj && (i >= 2 || j >= 2)) {
        const R zo = a.zout[p], gp = roms_gp<R, PH>(a, p, zo);
        const R fa = rmul(rmul(R(0.5), a.zrhs[p] + h[p]), g.fomn[p]);
        const R dk = a.zkstp[p] + h[p], dz = zo + h[p], ue = u[p + 1], vn = v[p + I];
        if (i >= 2) {
            const int w = p - 1;
            const R zw = a.zout[w], fw = rmul(rmul(R(0.5), a.zrhs[w] + h[w]), g.fomn[w]);
            const R cor = rfma(fa, v[p] + vn, rmul(fw, v[w] + v[w + I]));
            const R pmn2 = rmul(g.pm[p] + g.pm[w], g.pn[p] + g.pn[w]);
            const R v4 = rmul(R(0.25), ((v[p] + vn) + v[w]) + v[w + I]);
            const R ru = roms_rhs<R, false>(g.on_u[p], roms_gp<R, PH>(a, w, zw), gp, h[w], h[p], cor, u[p], v4, rdrag2,
                                            a.sustr[p], ddiv(R(4.0), pmn2));
            R f = ru;
            if (PH == 0) runew = ru;
            else if (!a.first) f = roms_am3(ru, a.ru_n[p], a.ru_b[p]);
            unew = roms_new(a.ukstp[p], dk + (a.zkstp[w] + h[w]), pmn2, cdt, f, dz + (zw + h[w]));
        }
        if (j >= 2) {
            const int q = p - I;
            const R zs = a.zout[q], fs = rmul(rmul(R(0.5), a.zrhs[q] + h[q]), g.fomn[q]);
            const R cor = rfma(fa, u[p] + ue, rmul(fs, u[q] + u[q + 1]));
            const R pmn2 = rmul(g.pm[p] + g.pm[q], g.pn[p] + g.pn[q]);
            const R u4 = rmul(R(0.25), ((u[p] + ue) + u[q]) + u[q + 1]);
            const R rv = roms_rhs<R, true>(g.om_v[p], roms_gp<R, PH>(a, q, zs), gp, h[q], h[p], cor, v[p], u4, rdrag2,
                                           a.svstr[p], ddiv(R(4.0), pmn2));
            R f = rv;
            if (PH == 0) rvnew = rv;
            else if (!a.first) f = roms_am3(rv, a.rv_n[p], a.rv_b[p]);
            vnew = roms_new(a.vkstp[p], dk + (a.zkstp[q] + h[q]), pmn2, cdt, f, dz + (zs + h[q]));
        }
    }
    a.uout[p] = unew;
    a.vout[p] = vnew;
    if (PH == 0) {
        a.ru_n[p] = runew;
        a.rv_n[p] = rvnew;
    }
}

// A copy of one value of the thread's own into its own shared-memory word: in flight without
// holding a register until it is read (after cp_own_wait).
template <typename T>
__device__ __forceinline__ void cp_own(T *dst, const T *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"((unsigned)__cvta_generic_to_shared(dst)),
                 "l"(src), "n"(sizeof(T))
                 : "memory");
}
__device__ __forceinline__ void cp_own_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int PENDING>
__device__ __forceinline__ void cp_own_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(PENDING) : "memory");
}

// A whole leapfrog / AM3 substep (predictor and corrector, free surface and momentum) in one launch.
// A block of 32 x H threads stages 32 columns (27 of them its own: lanes 3..29) and H rows (H - 3 its
// own: warps 2 .. H - 2), one node per thread.  Every node's inputs are loaded at once; the four
// stages then follow with x-neighbours by shuffle, y-neighbours through shared memory and three
// barriers, the halo nodes computing again what their owners compute.  Per substep and node 172
// bytes in FP32 (levels n and n-1, metrics, stresses and tendencies read once, level n+1 and the
// tendencies written, 80 bytes of FP64 averages) against 252 in two launches, and one launch
// latency, which is what small grids pay for.
//
// Level n+1 goes to the scratch slot (zout, uout, vout = slot p), because other blocks still read
// slot b at their halos; the host rotates the three slots.
template <typename R, int H, bool LATE>
__device__ __forceinline__ void roms_sub_tile(const Geo<R> &g, const RomsArgs<R> &a, const int i0,
                                              const int j0, unsigned char *raw) {
    const int I = g.I, J = g.J, lane = threadIdx.x & 31, wy = threadIdx.x >> 5;
    const int i = i0 - 3 + lane, j = j0 - 2 + wy;
    const int il = i < 0 ? 0 : (i > I - 1 ? I - 1 : i), jl = j < 0 ? 0 : (j > J - 1 ? J - 1 : j);
    const int js = j - 1 < 0 ? 0 : (j - 1 > J - 1 ? J - 1 : j - 1);
    const int jn = j + 1 < 0 ? 0 : (j + 1 > J - 1 ? J - 1 : j + 1);
    const int q = jl * I + il, qs = js * I + il, qn = jn * I + il;
    const bool ri = i >= 1 && i <= I - 2, rj = j >= 1 && j <= J - 2;
    const bool uface = i >= 2 && ri && rj, vface = j >= 2 && rj && ri;
    const bool mine = lane >= 3 && lane <= 29 && i < I && wy >= 2 && wy <= H - 2 && j < J;
    auto west = [](R x) { return __shfl_up_sync(0xffffffffu, x, 1); };
    auto east = [](R x) { return __shfl_down_sync(0xffffffffu, x, 1); };
    const R rdrag2 = (R)a.rdrag2, dt = (R)a.dtfast, dt2 = (R)(2.0 * a.dtfast), dth = (R)(0.5 * a.dtfast);
    // the context's metrics do not depend on the kernels before: loaded while those finish
    const R h = g.h[q], hs = g.h[qs], hn = g.h[qn], om = g.om_v[q], omN = g.om_v[qn];
    const R on = g.on_u[q], pm = g.pm[q], pn = g.pn[q], fo = g.fomn[q];
    pdl_enter();
    // LATE: values needed late wait in shared memory (averages; the old level's velocities, stresses,
    // tendencies), which leaves registers for more blocks per SM; else in registers
    constexpr int T = 32 * H;
    double *const av = reinterpret_cast<double *>(raw) + threadIdx.x;
    R *const own = reinterpret_cast<R *>(raw + 5 * T * sizeof(double)) + threadIdx.x;
    R *const sm = reinterpret_cast<R *>(raw + (LATE ? T * (5 * sizeof(double) + 7 * sizeof(R)) : 0)) + 32;
    // level n at the node and its row neighbours
    const R zn = a.zrhs[q], un = a.urhs[q], vn = a.vrhs[q];
    const R zs_ = a.zrhs[qs], zn_ = a.zrhs[qn], vN = a.vrhs[qn], zb = a.zkstp[q];
    const R *const lp[7] = {a.ukstp, a.vkstp, a.sustr, a.svstr, a.rz_b, a.ru_b, a.rv_b};
    double *const ap[5] = {a.Zt, a.DU1, a.DV1, a.DU2, a.DV2};
    enum { UB, VB, SU, SV, RZB, RUB, RVB };
    R lr[7];
    double ar[5];
#pragma unroll
    for (int f = 0; f < 7; ++f) {
        if constexpr (LATE) cp_own(own + f * T, lp[f] + q);
        else lr[f] = lp[f][q];
    }
    if constexpr (LATE) cp_own_commit();
    if (a.acc && mine) {
#pragma unroll
        for (int f = 0; f < 5; ++f) {
            if constexpr (LATE) cp_own(av + f * T, ap[f] + q);
            else ar[f] = ap[f][q];
        }
    }
    if constexpr (LATE) cp_own_commit();
    auto late = [&](int f) -> R {
        if constexpr (LATE) return own[f * T];
        else return lr[f];
    };
    auto avg = [&](int f) -> double {
        if constexpr (LATE) return av[f * T];
        else return ar[f];
    };
    constexpr int S = T;   // one exchanged field
    R *const me = sm + threadIdx.x;
    enum { GP, DK, VF, U, PM, PN, DZ, VP };
#define SF_SOUTH(f) me[(f) * S - 32]
#define SF_NORTH(f) me[(f) * S + 32]
    // rows 0 and H - 1 have no southern / northern neighbour in the block: what is then read lies in
    // the neighbouring field (or the pad before the first) and reaches no owned node
    // predictor: free surface
    const R D = zn + h, Ds = zs_ + hs, Dn = zn_ + hn;
    const R onE = east(on), pmn = rmul(pm, pn);
    const R au = rmul(un, rmul(R(0.5), D + west(D))), du = rmul(au, on);
    const R dv = rmul(rmul(vn, rmul(R(0.5), D + Ds)), om);
    const R dvN = rmul(rmul(vN, rmul(R(0.5), Dn + D)), omN);
    const R rz = rfma(-east(au), onE, du) + (dv - dvN);
    const R zp = rfma(rmul(pmn, dt2), rz, zb);
    R gp = rfma(R(0.68), zn, rmul(R(0.16), zb + zp));
    const R dk = zb + h, dz = zp + h, ue = east(un);
    R fa = rmul(rmul(R(0.5), D), fo), vf = rmul(fa, un + ue);
    me[GP * S] = gp;
    me[DK * S] = dk;
    me[VF * S] = vf;
    me[U * S] = un;
    me[PM * S] = pm;
    me[PN * S] = pn;
    me[DZ * S] = dz;
    __syncthreads();
    // predictor: momentum (not on row 0, nor U faces on row H - 1: no owned node needs them)
    if constexpr (LATE) cp_own_wait<1>();
    const R hw = west(h), pmw = rmul(pm + west(pm), pn + west(pn));
    const R pms = rmul(pm + SF_SOUTH(PM), pn + SF_SOUTH(PN));
    const R areaU = ddiv(R(4.0), pmw), areaV = ddiv(R(4.0), pms);
    R up = R(0), vp = R(0), ru = R(0), rv = R(0);
    if (wy > 0) {
        const R gw = west(gp), cor = rfma(fa, vn + vN, west(rmul(fa, vn + vN)));
        const R v4 = rmul(R(0.25), ((vn + vN) + west(vn)) + west(vN));
        const R dkw = dk + west(dk), dzw = dz + west(dz);
        if (uface && wy < H - 1) {
            ru = roms_rhs<R, false>(on, gw, gp, hw, h, cor, un, v4, rdrag2, late(SU), areaU);
            up = roms_new(late(UB), dkw, pmw, dt, ru, dzw);
        }
        if (vface) {
            const R u4 = rmul(R(0.25), ((un + ue) + SF_SOUTH(U)) + me[U * S - 31]);
            rv = roms_rhs<R, true>(om, SF_SOUTH(GP), gp, hs, h, rfma(fa, un + ue, SF_SOUTH(VF)), vn, u4,
                                   rdrag2, late(SV), areaV);
            vp = roms_new(late(VB), dk + SF_SOUTH(DK), pms, dt, rv, dz + SF_SOUTH(DZ));
        }
    }
    me[VP * S] = vp;
    __syncthreads();
    // corrector: free surface (rows 1 .. H - 2)
    R vpN = R(0), upE = R(0), dup = R(0), dvp = R(0), zc = R(0), dzc = R(0);
    if (wy > 0 && wy < H - 1) {
        vpN = SF_NORTH(VP);
        upE = east(up);
        const R aup = rmul(up, rmul(R(0.5), dz + west(dz)));
        dup = rmul(aup, on);
        dvp = rmul(rmul(vp, rmul(R(0.5), dz + SF_SOUTH(DZ))), om);
        const R dvpN = rmul(rmul(vpN, rmul(R(0.5), SF_NORTH(DZ) + dz)), omN);
        const R rzc = rfma(-east(aup), onE, dup) + (dvp - dvpN);
        zc = rfma(rmul(pmn, dt), roms_am3(rzc, rz, late(RZB)), zn);
        gp = rfma(R(0.6), zc, rmul(R(0.4), zp));
        dzc = zc + h;
        fa = rmul(rmul(R(0.5), dz), fo);
        vf = rmul(fa, up + upE);
        me[GP * S] = gp;   // the predictor's values of these fields were read before the last barrier
        me[DK * S] = dzc;
        me[VF * S] = vf;
        me[U * S] = up;
    }
    __syncthreads();
    if (wy < 2 || wy > H - 2) return;
    // corrector: momentum (the owned rows)
    R uc = R(0), vc = R(0);
    {
        const R gw = west(gp), cor = rfma(fa, vp + vpN, west(rmul(fa, vp + vpN)));
        const R v4 = rmul(R(0.25), ((vp + vpN) + west(vp)) + west(vpN));
        const R Dw = D + west(D), dzw = dzc + west(dzc);
        if (uface) {
            const R r = roms_rhs<R, false>(on, gw, gp, hw, h, cor, up, v4, rdrag2, late(SU), areaU);
            uc = roms_new(un, Dw, pmw, dth, roms_am3(r, ru, late(RUB)), dzw);
        }
        if (vface) {
            const R u4 = rmul(R(0.25), ((up + upE) + SF_SOUTH(U)) + me[U * S - 31]);
            const R r = roms_rhs<R, true>(om, SF_SOUTH(GP), gp, hs, h, rfma(fa, up + upE, SF_SOUTH(VF)), vp, u4,
                                          rdrag2, late(SV), areaV);
            vc = roms_new(vn, D + Ds, pms, dth, roms_am3(r, rv, late(RVB)), dzc + SF_SOUTH(DK));
        }
    }
#undef SF_SOUTH
#undef SF_NORTH
    if (!mine) return;
    a.uout[q] = uc;
    a.vout[q] = vc;
    a.ru_n[q] = ru;
    a.rv_n[q] = rv;
    a.rz_n[q] = ri && rj ? rz : R(0);
    if (ri && rj) {   // the free surface, and the ring nodes next to it
        const int di = i == 1 ? -1 : (i == I - 2 ? 1 : 0), dj = j == 1 ? -I : (j == J - 2 ? I : 0);
        a.zout[q] = zc;
        if (di) a.zout[q + di] = zc;
        if (dj) a.zout[q + dj] = zc;
        if (di && dj) a.zout[q + di + dj] = zc;
    }
    if (a.acc) {
        if constexpr (LATE) cp_own_wait<0>();
        const double un1 = i < 1 ? 0.0 : (double)du, vn1 = j < 1 ? 0.0 : (double)dv;
        const double up1 = i < 1 ? 0.0 : (double)dup, vp1 = j < 1 ? 0.0 : (double)dvp;
        a.Zt[q] = rsum<R>(avg(0), a.c1, (double)zn);
        a.DU1[q] = rsum<R>(avg(1), a.c1, un1);
        a.DV1[q] = rsum<R>(avg(2), a.c1, vn1);
        a.DU2[q] = rsum<R>(rsum<R>(avg(3), a.c2, un1), a.c2c, up1);
        a.DV2[q] = rsum<R>(rsum<R>(avg(4), a.c2, vn1), a.c2c, vp1);
    }
}

// The fast-time averages of the loop's last substep (nfast + 1), which only accumulates the fields
// of level n (step2d_LF_AM3.h.py:923-926).
template <typename R>
__device__ __forceinline__ void roms_acc_at(const Geo<R> &g, const RomsArgs<R> &a, const long p) {
    if (p >= g.s2) return;
    const int j = fdiv((int)p, g.dI), i = (int)p - j * g.I;
    const R *z = a.zrhs, *h = g.h;
    const R D = z[p] + h[p];
    double du = 0.0, dv = 0.0;
    if (i >= 1) du = (double)rmul(rmul(a.urhs[p], rmul(R(0.5), D + (z[p - 1] + h[p - 1]))), g.on_u[p]);
    if (j >= 1) dv = (double)rmul(rmul(a.vrhs[p], rmul(R(0.5), D + (z[p - g.I] + h[p - g.I]))), g.om_v[p]);
    a.Zt[p] = rsum<R>(a.Zt[p], a.c1, (double)z[p]);
    a.DU1[p] = rsum<R>(a.DU1[p], a.c1, du);
    a.DV1[p] = rsum<R>(a.DV1[p], a.c1, dv);
    a.DU2[p] = rsum<R>(a.DU2[p], a.c2, du);
    a.DV2[p] = rsum<R>(a.DV2[p], a.c2, dv);
}

// The ROMS-form 3D momentum right-hand side at the interior faces (U: j = 1..J-2, i = 2..I-2;
// V: j = 2..J-2, i = 1..I-2), 0 elsewhere, every level: Coriolis as ROMS's (and the
// reference's addCoriolis), then second-order centred advection of momentum: horizontal
// fluxes UFx = (Huon_i + Huon_i+1)/4 (u_i + u_i+1) at rho points and UFe = (Hvom_i +
// Hvom_i-1)/4 (u_j + u_j-1) at psi points (the UV_C2ADVECTION form of the reference's ROMS
// transcription, obsolete/step2d_LF_AM3.h.py:1244-1300, per level), V alike; the vertical
// advection is implicit, in the column solve (roms_column).  The expressions keep the oracle's
// operand order (oracle/roms_oracle.py, rhs3d).
//
// A warp takes a strip of 29 columns (lanes 1 .. 29; 0 and 30 their neighbours) of one level and
// walks up its rows: every field is loaded once per node, west and east by shuffle, the southern
// fluxes from the row before, the next row's loads in flight.  Bound: the 28 bytes a point and level
// in FP32 (0.45 ms for 2050 x 1026 x 50 at the copy bandwidth); a thread per column loading some 25
// neighbour values a level took 1.19 ms.
template <typename R>
struct RhsRow {
    R u, v, hu, hv, hz, fo;
};
template <typename R>
__device__ __forceinline__ void roms_rhs3d_rows(const Geo<R> &g, const R *__restrict__ u,
                                                const R *__restrict__ v, const R *__restrict__ Hu,
                                                const R *__restrict__ Hv, const R *__restrict__ Hz,
                                                R *__restrict__ ru, R *__restrict__ rv, const int i0,
                                                const int j0, const int nrows, const int k) {
    const int I = g.I, J = g.J, lane = threadIdx.x & 31;
    if (j0 >= J) return;   // whole warp
    const int i = i0 - 1 + lane, il = i < 0 ? 0 : (i > I - 1 ? I - 1 : i);
    const bool out = lane >= 1 && lane <= kRomsCols && i < I;
    const int jend = j0 + nrows < J ? j0 + nrows : J;
    const long o = (long)k * g.s2;
    if (k >= g.N) {   // the level above the surface
        if (out)
            for (int j = j0; j < jend; ++j) {
                ru[o + j * I + i] = R(0);
                rv[o + j * I + i] = R(0);
            }
        return;
    }
    u += o;
    v += o;
    Hu += o;
    Hv += o;
    Hz += o;
    ru += o;
    rv += o;
    auto west = [](R x) { return __shfl_up_sync(0xffffffffu, x, 1); };
    auto east = [](R x) { return __shfl_down_sync(0xffffffffu, x, 1); };
    auto load = [&](int j) {
        const int p = (j < 0 ? 0 : (j > J - 1 ? J - 1 : j)) * I + il;
        return RhsRow<R>{u[p], v[p], Hu[p], Hv[p], Hz[p], g.fomn[p]};
    };
    RhsRow<R> c = load(j0 - 1), n = load(j0);
    R hus = R(0), es = R(0), vfs = R(0), eps = R(0);   // the row below: Hu, its northern fluxes
    for (int j = j0 - 1; j < jend; ++j) {
        const RhsRow<R> nn = load(j + 2);   // in flight
        const R ue = east(c.u), vw = west(c.v);
        // factors of the Coriolis terms and of the momentum fluxes; differences and sums of two products
        // with the contraction written out (rfma)
        const R cf = rmul(c.hz, c.fo), vb = rmul(c.v + n.v, R(0.5)), ub = rmul(c.u + ue, R(0.5));
        const R vf = rmul(cf, ub);
        const R hu = rmul(R(0.25), c.hu + east(c.hu)), wu = c.u + ue;           // at rho points
        const R hn = rmul(R(0.25), n.hv + west(n.hv)), yn = n.u + c.u, en = rmul(hn, yn);   // at psi points
        const R hx = rmul(R(0.25), c.hu + hus), wx = c.v + vw, xv = rmul(hx, wx);
        const R hp = rmul(R(0.25), c.hv + n.hv), yp = c.v + n.v, ep = rmul(hp, yp);
        const R ufw = west(rmul(cf, vb)), xuw = west(rmul(hu, wu)), hxe = east(hx), wxe = east(wx);
        if (j >= j0 && out) {
            R tu = R(0), tv = R(0);
            if (i >= 2 && i <= I - 2 && j >= 1 && j <= J - 2)
                tu = rmul(rfma(cf, vb, ufw), R(0.5)) - (rfma(hu, wu, -xuw) + rfma(hn, yn, -es));
            if (j >= 2 && j <= J - 2 && i >= 1 && i <= I - 2)
                tv = -rmul(rfma(cf, ub, vfs), R(0.5)) - (rfma(hxe, wxe, -xv) + rfma(hp, yp, -eps));
            ru[j * I + i] = tu;
            rv[j * I + i] = tv;
        }
        es = en;
        vfs = vf;
        eps = ep;
        hus = c.hu;
        c = n;
        n = nn;
    }
}

// The same, a point a thread, levels k0, k0 + dk, ..., every neighbour loaded where it is needed: for basins whose
// strips would be mostly empty (rule: Ops::roms_rhs3d).  U and V in branches of their own, loads they share
// included: in one branch 5 x 200000 points of 5 levels in FP32 took 100 us, so 48.
template <typename R>
__device__ __forceinline__ void roms_rhs3d_point(const Geo<R> &g, const R *__restrict__ u, const R *__restrict__ v,
                                                 const R *__restrict__ Hu, const R *__restrict__ Hv,
                                                 const R *__restrict__ Hz, R *__restrict__ ru, R *__restrict__ rv,
                                                 const long p, const int k0, const int dk) {
    if (p >= g.s2) return;
    const int j = fdiv((int)p, g.dI), i = (int)p - j * g.I;
    const long I = g.I, s2 = g.s2;
    const int N = g.N;
    const bool uf = i >= 2 && i <= g.I - 2 && j >= 1 && j <= g.J - 2;
    const bool vf = j >= 2 && j <= g.J - 2 && i >= 1 && i <= g.I - 2;
    const R *fo = g.fomn;
    for (int k = k0; k <= N; k += dk) {
        const long o = (long)k * s2;
        R tu = R(0), tv = R(0);
        if (k < N && uf) {
            const R *uk = u + o, *vk = v + o, *hu = Hu + o, *hv = Hv + o, *hz = Hz + o;
            const R cf = rmul(hz[p], fo[p]), vb = rmul(vk[p] + vk[p + I], R(0.5));
            const R ufw = rmul(rmul(hz[p - 1], fo[p - 1]), rmul(vk[p - 1] + vk[p - 1 + I], R(0.5)));
            const R xuw = rmul(rmul(R(0.25), hu[p - 1] + hu[p]), uk[p - 1] + uk[p]);
            const R es = rmul(rmul(R(0.25), hv[p] + hv[p - 1]), uk[p] + uk[p - I]);
            tu = rmul(rfma(cf, vb, ufw), R(0.5)) - (rfma(rmul(R(0.25), hu[p] + hu[p + 1]), uk[p] + uk[p + 1], -xuw) +
                                                    rfma(rmul(R(0.25), hv[p + I] + hv[p + I - 1]), uk[p + I] + uk[p], -es));
        }
        if (k < N && vf) {
            const R *uk = u + o, *vk = v + o, *hu = Hu + o, *hv = Hv + o, *hz = Hz + o;
            const R cf = rmul(hz[p], fo[p]), ub = rmul(uk[p] + uk[p + 1], R(0.5));
            const R vfs = rmul(rmul(hz[p - I], fo[p - I]), rmul(uk[p - I] + uk[p - I + 1], R(0.5)));
            const R xv = rmul(rmul(R(0.25), hu[p] + hu[p - I]), vk[p] + vk[p - 1]);
            const R eps = rmul(rmul(R(0.25), hv[p - I] + hv[p]), vk[p - I] + vk[p]);
            tv = -rmul(rfma(cf, ub, vfs), R(0.5)) - (rfma(rmul(R(0.25), hu[p + 1] + hu[p + 1 - I]), vk[p + 1] + vk[p], -xv) +
                                                     rfma(rmul(R(0.25), hv[p] + hv[p + I]), vk[p] + vk[p + I], -eps));
        }
        ru[o + p] = tu;
        rv[o + p] = tv;
    }
}

// Surface and bottom stress on the 3D momentum right-hand side (ROMS's ru includes
// + sustr om_u on_u at k = N and - bustr om_u on_u at k = 1): ru[N-1] += sustr * area and
// ru[0] -= rdrag2 ub sqrt(ub^2 + v_u^2) * area at the interior U faces, ub the bottom level's u,
// v_u the four-point average of its v; rv likewise at the interior V faces.
template <typename R>
__device__ __forceinline__ void roms_stress3d_at(const Geo<R> &g, const R *__restrict__ u,
                                                 const R *__restrict__ v, R *__restrict__ ru,
                                                 R *__restrict__ rv, const R *__restrict__ sustr,
                                                 const R *__restrict__ svstr, R rdrag2,
                                                 const long p) {
    if (p >= g.s2) return;
    const int j = fdiv((int)p, g.dI), i = (int)p - j * g.I;
    const long I = g.I, o = (long)(g.N - 1) * g.s2 + p;
    if (i >= 2 && i <= g.I - 2 && j >= 1 && j <= g.J - 2) {
        const R area = ddiv(R(4.0), (g.pm[p] + g.pm[p - 1]) * (g.pn[p] + g.pn[p - 1]));
        const R v4 = R(0.25) * (((v[p] + v[p + I]) + v[p - 1]) + v[p + I - 1]);
        const R ub = u[p];
        const R bustr = rdrag2 * ub * sqrt(ub * ub + v4 * v4);
        ru[o] = ru[o] + sustr[p] * area;
        ru[p] = ru[p] - bustr * area;
    }
    if (j >= 2 && j <= g.J - 2 && i >= 1 && i <= g.I - 2) {
        const R area = ddiv(R(4.0), (g.pm[p] + g.pm[p - I]) * (g.pn[p] + g.pn[p - I]));
        const R u4 = R(0.25) * (((u[p] + u[p + 1]) + u[p - I]) + u[p - I + 1]);
        const R vb = v[p];
        const R bvstr = rdrag2 * vb * sqrt(u4 * u4 + vb * vb);
        rv[o] = rv[o] + svstr[p] * area;
        rv[p] = rv[p] - bvstr * area;
    }
}

// The ROMS-form step3d_uv for one face column (d = 1: U face, d = I: V face): with F_w the
// upwind vertical advective flux through w level w (w_w x_w-1 where w_w > 0, w_w x_w where
// w_w < 0; w_w = fac (W_w + W_w,nbr) / 2, 0 at the bottom and the surface), fac = dt pmU pnU,
//   Hzu_k x_k - [viscosity] + (F_k+1 - F_k) = Hzu_k u_k + fac r_k,
// r_k = (c0 ru_k(n) + c1 ru_k(n-1)) + c2 ru_k(n-2) (Adams-Bashforth), the viscosity through
// FC_k = -lamdt AKU_k+1 / DZ_k on the interface between levels k and k+1 (w level k+1; no flux
// through the surface or the bottom, whose stresses are in ru): the lower, main and upper
// diagonals l_k = FC_k-1 - w+_k, b_k = (Hzu_k - FC_k - FC_k-1) + (w+_k+1 - w-_k),
// u_k = FC_k + w-_k+1 (an M-matrix at any vertical Courant number: backward-Euler upwind
// vertical advection).  Thomas elimination in R, then the depth mean set to the barotropic
// transport with FP64 sums: x_k -= (sum Hzu x - avg/on) / sum Hzu.  Returns the new depth-mean
// velocity avg/on/sum Hzu.
// Bound: latency of the level loads at 12 to 16 warps per SM (56 bytes a point and component pair in
// FP32, 1.4 GB and 0.21 ms at the copy bandwidth for 1003 x 501 x 50; 0.82 ms before with per-thread
// local arrays and U and V columns half a grid apart, 0.45 now).
template <typename R>
struct RomsRhs {
    const R *r0, *r1, *r2;   // right-hand sides at n, n-1, n-2
};

// Levels whose loads the column solve issues together (1003 x 501 x 50, FP32: 2, 4, 6, 8, 12 levels 0.59,
// 0.59, 0.47, 0.45, 0.53 ms; FP64 4, 6, 8: 1.29, 1.27, 1.33), and the blocks per SM its registers are capped
// for.  Columns of at most 16 levels (SHORT) have few chunks to issue and little shared memory, so more blocks
// hide the latency instead: 1026 x 514 x 6 in FP32 104 us with 8 levels and 3 blocks, 66 with 2 and 8, FP64 189 and
// 112 (2 and 10); 16 levels FP32 188 and 128, FP64 361 and 249; at 24 levels the long form leads (FP32 255
// against 282 us).
constexpr int kRomsShortN = 16;
template <typename R>
constexpr int roms_col_chunk(bool SHORT) { return SHORT ? 2 : (sizeof(R) == 4 ? 8 : 6); }
template <typename R>
constexpr int roms_col_blocks(bool SHORT) { return !SHORT ? 3 : (sizeof(R) == 4 ? 8 : 10); }
// A pivot of the elimination as its divisions use it: in FP32 the reciprocal (a / b through
// __fdividef is a times the hardware reciprocal of b, bit for bit in b's normal range, and every
// pivot divides twice), in FP64 the pivot itself (IEEE division).
__device__ __forceinline__ float roms_pivot(float b) {
    float r;
    asm("rcp.approx.f32 %0, %1;" : "=f"(r) : "f"(b));
    return r;
}
__device__ __forceinline__ double roms_pivot(double b) { return b; }
__device__ __forceinline__ float over_pivot(float a, float r) { return __fmul_rn(a, r); }
__device__ __forceinline__ double over_pivot(double a, double b) { return a / b; }
// a / b, its last product not fused into a sum that takes it
template <typename R>
__device__ __forceinline__ R roms_div(R a, R b) { return over_pivot(a, roms_pivot(b)); }

// Per column two arrays in shared memory, [level][thread]: the pivots, overwritten by the solution, and
// the upper diagonals; the eliminated right-hand side takes the column's own place in u until the
// solution does.  Levels are taken in whole chunks whose loads are issued together, then one by
// one: a test per level inside a chunk (the level below N?) cost some 300 cycles a level.
// Off: element offsets in a field (32-bit where they fit).
template <typename R, int T, typename Off, bool SHORT>
__device__ __forceinline__ double roms_column(const Geo<R> &g, const int p, const int d, R *__restrict__ u,
                                              RomsRhs<R> rs, R c0, R c1, R c2, const R *__restrict__ Hz,
                                              const R *__restrict__ Akv, const R *__restrict__ z_r,
                                              const R *__restrict__ W, double avg, R on, R dt, R lamdt,
                                              R *__restrict__ col) {
    const Off s2 = (Off)g.s2;
    const int N = g.N;
    const R pmU = rmul(R(0.5), g.pm[p] + g.pm[p - d]);
    const R pnU = rmul(R(0.5), g.pn[p] + g.pn[p - d]);
    const R fac = rmul(dt, rmul(pmU, pnU));
    auto wplus = [](R w) { return w > R(0) ? w : R(0); };
    auto wminus = [](R w) { return w < R(0) ? w : R(0); };
    R fcm = R(0), wk = R(0);   // FC of the level below, the flux through this level's bottom
    R pv = R(1), upp = R(0), xp = R(0);   // the level below's eliminated row (none: w = 0 / 1)
    R zr = z_r[p], zq = z_r[p - d];       // z_r of the level in hand, both rho points
    double H = 0.0;
    R *bu = col;                          // the level's pivot, upper diagonal at bu[T]
    Off o = (Off)p;
    // elimination of a level: its FC and the flux through its top are given (0 at the surface)
    auto eliminate = [&](R hza, R hzb, R fck, R wk1, R q0, R q1, R q2, R uo) {
        const R hzu = rmul(R(0.5), hza + hzb);
        R b = ((hzu - fck) - fcm) + (wplus(wk1) - wminus(wk));
        const R upk = fck + wminus(wk1);
        const R r = rfma(c2, q2, rfma(c0, q0, rmul(c1, q1)));
        R x = rfma(hzu, uo, rmul(fac, r));
        const R w = over_pivot(fcm - wplus(wk), pv);
        b = rfma(-w, upp, b);
        x = rfma(-w, xp, x);
        pv = roms_pivot(b);
        bu[0] = pv;
        bu[T] = upk;
        bu += 2 * T;
        u[o] = x;
        o += s2;
        H = H + (double)hzu;
        upp = upk;
        xp = x;
        fcm = fck;
        wk = wk1;
    };
    auto levels = [&](auto n) {   // levels below the surface one
        constexpr int C = decltype(n)::value;
        R hz0[C], hz1[C], ak0[C], ak1[C], zr0[C], zq0[C], w0[C], w1[C], q0[C], q1[C], q2[C], uo[C];
        Off l = o;
#pragma unroll
        for (int c = 0; c < C; ++c, l += s2) {
            const Off t = l + s2;
            hz0[c] = Hz[l];
            hz1[c] = Hz[l - d];
            ak0[c] = Akv[t];
            ak1[c] = Akv[t - d];
            zr0[c] = z_r[t];
            zq0[c] = z_r[t - d];
            w0[c] = W[t];
            w1[c] = W[t - d];
            q0[c] = rs.r0[l];
            q1[c] = rs.r1[l];
            q2[c] = rs.r2[l];
            uo[c] = u[l];
        }
#pragma unroll
        for (int c = 0; c < C; ++c) {
            const R ak = rmul(R(0.5), ak0[c] + ak1[c]);
            const R dz = rmul(R(0.5), (zr0[c] - zr) + (zq0[c] - zq));
            zr = zr0[c];
            zq = zq0[c];
            eliminate(hz0[c], hz1[c], roms_div(rmul(-lamdt, ak), dz), rmul(fac, rmul(R(0.5), w0[c] + w1[c])), q0[c],
                      q1[c], q2[c], uo[c]);
        }
    };
    in_chunks<roms_col_chunk<R>(SHORT)>(N - 1, levels);
    eliminate(Hz[o], Hz[o - d], R(0), R(0), rs.r0[o], rs.r1[o], rs.r2[o], u[o]);
    // back substitution
    R x = over_pivot(xp, pv);
    bu -= 2 * T;
    bu[0] = x;
    o -= s2;
    auto back = [&](auto n) {
        constexpr int C = decltype(n)::value;
        R q[C], pk[C], uk[C];
#pragma unroll
        for (int c = 0; c < C; ++c) {
            o -= s2;
            q[c] = u[o];
            pk[c] = bu[-2 * T * (c + 1)];
            uk[c] = bu[-2 * T * (c + 1) + T];
        }
#pragma unroll
        for (int c = 0; c < C; ++c) {
            bu -= 2 * T;
            x = over_pivot(rfma(-uk[c], x, q[c]), pk[c]);
            bu[0] = x;
        }
    };
    in_chunks<8>(N - 1, back);
    double Hu = 0.0;
    o = (Off)p;
#pragma unroll 8
    for (int k = 0; k < N; ++k, o += s2)
        Hu = rsum<R>(Hu, (double)rmul(R(0.5), Hz[o] + Hz[o - d]), (double)col[k * (2 * T)]);
    const double target = avg / (double)on;
    const double udiff = (Hu - target) / H;
    o = (Off)p;
#pragma unroll 8
    for (int k = 0; k < N; ++k, o += s2) u[o] = (R)((double)col[k * (2 * T)] - udiff);
    return target / H;
}

// Threads per block of the column solve: 2 N values of shared memory per thread.
template <typename R>
constexpr int roms_col_threads() { return sizeof(R) == 4 ? 128 : 64; }

// The ROMS-form step3d_uv over the interior faces (U: j = 1..J-2, i = 2..I-2; V: j = 2..J-2,
// i = 1..I-2), one thread per face column: the U column (west face) or the V column (south face,
// vcol) of rho point p; and the barotropic restart: ubar, vbar in slots n and scratch = the new
// depth-mean velocities at those faces, 0 elsewhere.
template <typename R, int T, typename Off, bool SHORT>
__device__ __forceinline__ void roms_step3d_at(const Geo<R> &g, R *__restrict__ u,
                                               R *__restrict__ v, RomsRhs<R> ru, RomsRhs<R> rv,
                                               R c0, R c1, R c2, R *__restrict__ ubar_n,
                                               R *__restrict__ vbar_n, R *__restrict__ ubar_s,
                                               R *__restrict__ vbar_s, const R *__restrict__ Hz,
                                               const R *__restrict__ Akv,
                                               const R *__restrict__ z_r,
                                               const R *__restrict__ W,
                                               const double *__restrict__ DU,
                                               const double *__restrict__ DV, R dt, R lamdt,
                                               const long t, const bool vcol, R *col) {
    if (t >= g.s2) return;
    const int p = (int)t, j = fdiv(p, g.dI), i = p - j * g.I;
    R bar = R(0);
    if (!vcol) {
        if (i >= 2 && i <= g.I - 2 && j >= 1 && j <= g.J - 2)
            bar = (R)roms_column<R, T, Off, SHORT>(g, p, 1, u, ru, c0, c1, c2, Hz, Akv, z_r, W, DU[p], g.on_u[p], dt,
                                       lamdt, col);
        ubar_n[p] = bar;
        ubar_s[p] = bar;
    } else {
        if (j >= 2 && j <= g.J - 2 && i >= 1 && i <= g.I - 2)
            bar = (R)roms_column<R, T, Off, SHORT>(g, p, g.I, v, rv, c0, c1, c2, Hz, Akv, z_r, W, DV[p], g.om_v[p],
                                       dt, lamdt, col);
        vbar_n[p] = bar;
        vbar_s[p] = bar;
    }
}

// Closed walls for the 3D velocities: u = 0 on the U wall faces (i = 1, I-1), v = 0 on the V
// wall faces (j = 1, J-1), every level.
template <typename R>
__device__ __forceinline__ void roms_walls3d_at(const Geo<R> &g, R *__restrict__ u,
                                                R *__restrict__ v, const long p) {
    if (p >= g.s2) return;
    const int j = fdiv((int)p, g.dI), i = (int)p - j * g.I;
    const bool uw = (i == 1 || i == g.I - 1), vw = (j == 1 || j == g.J - 1);
    if (!uw && !vw) return;
    for (int k = 0; k <= g.N; ++k) {
        if (uw) u[(long)k * g.s2 + p] = R(0);
        if (vw) v[(long)k * g.s2 + p] = R(0);
    }
}

// Kernels: a single grid (one thread per flat point) and ensembles (a block map gives each
// block its member and its block within the member; the member's fields are offset in the
// pools: 2D fields by off2, fields of N+1 levels by off3, of N levels by offN).
template <typename R>
struct MemberAt {
    Geo<R> g;
    long o2, o3, oN, p;
};
template <typename R>
__device__ __forceinline__ MemberAt<R> member_at(const Member<R> *mt, const int2 *bm, int bs) {
    const int2 mb = bm[blockIdx.x];
    const Member<R> &M = mt[mb.x];
    return MemberAt<R>{M.g, M.off2, M.off3, M.offN, (long)mb.y * bs + threadIdx.x};
}
template <typename T>
__device__ __forceinline__ T *at(T *x, long o) { return x ? x + o : x; }
template <typename R>
__device__ __forceinline__ RomsArgs<R> roms_args_at(const RomsArgs<R> &a, long o) {
    RomsArgs<R> b = a;
    b.zrhs = at(a.zrhs, o); b.urhs = at(a.urhs, o); b.vrhs = at(a.vrhs, o);
    b.zkstp = at(a.zkstp, o); b.ukstp = at(a.ukstp, o); b.vkstp = at(a.vkstp, o);
    b.zout = at(a.zout, o); b.uout = at(a.uout, o); b.vout = at(a.vout, o);
    b.rz_n = at(a.rz_n, o); b.ru_n = at(a.ru_n, o); b.rv_n = at(a.rv_n, o);
    b.rz_b = at(a.rz_b, o); b.ru_b = at(a.ru_b, o); b.rv_b = at(a.rv_b, o);
    b.sustr = at(a.sustr, o); b.svstr = at(a.svstr, o);
    b.Zt = at(a.Zt, o); b.DU1 = at(a.DU1, o); b.DV1 = at(a.DV1, o);
    b.DU2 = at(a.DU2, o); b.DV2 = at(a.DV2, o);
    return b;
}

template <typename R, int PH>
__global__ void __launch_bounds__(32 * kRomsWarps) k_roms_phase(Geo<R> g, RomsArgs<R> a, int nrows) {
    pdl_enter();
    roms_phase_rows<R, PH>(g, a, (int)blockIdx.x * kRomsCols,
                           ((int)blockIdx.y * kRomsWarps + (int)(threadIdx.x >> 5)) * nrows, nrows);
}
template <typename R, int PH>
__global__ void __launch_bounds__(32 * kRomsWarps) kb_roms_phase(const Member<R> *mt, const int2 *bm,
                                                                 RomsArgs<R> a, int nrows) {
    pdl_enter();
    const int2 mb = bm[blockIdx.x];
    const Member<R> &M = mt[mb.x];
    const int ns = (M.g.I + kRomsCols - 1) / kRomsCols, by = mb.y / ns, bx = mb.y - by * ns;
    roms_phase_rows<R, PH>(M.g, roms_args_at(a, M.off2), bx * kRomsCols,
                           (by * kRomsWarps + (int)(threadIdx.x >> 5)) * nrows, nrows);
}
template <typename R, int PH, bool MOM>
__global__ void __launch_bounds__(256) k_roms_point(Geo<R> g, RomsArgs<R> a) {
    pdl_enter();
    if constexpr (MOM) roms_mom_point<R, PH>(g, a, tid_flat());
    else roms_zeta_point<R, PH>(g, a, tid_flat());
}
template <typename R, int PH, bool MOM>
__global__ void __launch_bounds__(256) kb_roms_point(const Member<R> *mt, const int2 *bm, RomsArgs<R> a) {
    pdl_enter();
    const MemberAt<R> m = member_at(mt, bm, 256);
    if constexpr (MOM) roms_mom_point<R, PH>(m.g, roms_args_at(a, m.o2), m.p);
    else roms_zeta_point<R, PH>(m.g, roms_args_at(a, m.o2), m.p);
}
// Shared memory of a block: per node (LATE) 5 averages and 7 late inputs, 8 exchanged values, and a
// row of pad on either side of the exchanged fields.
template <typename R, bool LATE>
constexpr int roms_sub_smem(int H) {
    return (LATE ? 32 * H * (40 + 7 * (int)sizeof(R)) : 0) + (8 * H + 2) * 32 * (int)sizeof(R);
}
// Blocks per SM the register cap allows for: LATE in FP32 3 of 384 threads at 56 registers (4 at 40
// spill: 2050 x 1026 loop 5.10 against 4.35 ms), in FP64 2 at 80 (68 bytes spilled); else uncapped.
template <typename R, bool LATE>
constexpr int roms_sub_blocks() { return !LATE ? 1 : (sizeof(R) == 4 ? 3 : 2); }
template <typename R, int H, bool LATE>
__global__ void __launch_bounds__(32 * H, roms_sub_blocks<R, LATE>()) k_roms_sub(Geo<R> g, RomsArgs<R> a) {
    extern __shared__ __align__(16) unsigned char sub_smem[];
    // grid.z: 65,535 rows of tiles each, past the end no node is owned
    roms_sub_tile<R, H, LATE>(g, a, (int)blockIdx.x * kSubCols, (int)(blockIdx.z * gridDim.y + blockIdx.y) * (H - 3),
                              sub_smem);
}
template <typename R, int H, bool LATE>
__global__ void __launch_bounds__(32 * H, roms_sub_blocks<R, LATE>()) kb_roms_sub(const Member<R> *mt, const int2 *bm,
                                                                               RomsArgs<R> a) {
    extern __shared__ __align__(16) unsigned char sub_smem[];
    const int2 mb = bm[blockIdx.x];
    const Member<R> &M = mt[mb.x];
    const int ns = (M.g.I + kSubCols - 1) / kSubCols, by = mb.y / ns, bx = mb.y - by * ns;
    roms_sub_tile<R, H, LATE>(M.g, roms_args_at(a, M.off2), bx * kSubCols, by * (H - 3), sub_smem);
}
template <typename R, bool LATE>
cudaError_t roms_sub_launch(const sf_ctx *c, const RomsArgs<R> &a, dim3 grid, cudaStream_t s) {
    constexpr int H = kSubRows, smem = roms_sub_smem<R, LATE>(H);
    static bool done[64] = {};   // the raised shared-memory limit, once on each device
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= 64 || !done[dev]) {
        const auto at = cudaFuncAttributeMaxDynamicSharedMemorySize;
        e = cudaFuncSetAttribute(k_roms_sub<R, H, LATE>, at, smem);
        if (e == cudaSuccess) e = cudaFuncSetAttribute(kb_roms_sub<R, H, LATE>, at, smem);
        if (e != cudaSuccess) return e;
        if (dev >= 0 && dev < 64) done[dev] = true;
    }
    if (c->nmem > 1)
        return launch_dep(c, kb_roms_sub<R, H, LATE>, grid, 32 * H, smem, s, mt<R>(c), c->bm_sub, a);
    return launch_dep(c, k_roms_sub<R, H, LATE>, grid, 32 * H, smem, s, Ops<R>::geo(c), a);
}
template <typename R>
__global__ void __launch_bounds__(256) k_roms_acc(Geo<R> g, RomsArgs<R> a) {
    pdl_enter();
    roms_acc_at(g, a, tid_flat());
}
template <typename R>
__global__ void __launch_bounds__(256) kb_roms_acc(const Member<R> *mt, const int2 *bm, RomsArgs<R> a) {
    pdl_enter();
    const MemberAt<R> m = member_at(mt, bm, 256);
    roms_acc_at(m.g, roms_args_at(a, m.o2), m.p);
}
template <typename R>
__global__ void __launch_bounds__(32 * kRomsWarps) k_roms_rhs3d(Geo<R> g, const R *u, const R *v, const R *Hu,
                                                                const R *Hv, const R *Hz, R *ru, R *rv,
                                                                int nrows) {
    roms_rhs3d_rows(g, u, v, Hu, Hv, Hz, ru, rv, (int)blockIdx.x * kRomsCols,
                    ((int)blockIdx.y * kRomsWarps + (int)(threadIdx.x >> 5)) * nrows, nrows, (int)blockIdx.z);
}
template <typename R>
__global__ void __launch_bounds__(32 * kRomsWarps) kb_roms_rhs3d(const Member<R> *mt, const int2 *bm, const R *u,
                                                                 const R *v, const R *Hu, const R *Hv,
                                                                 const R *Hz, R *ru, R *rv, int nrows) {
    const int2 mb = bm[blockIdx.x];
    const Member<R> &M = mt[mb.x];
    if ((int)blockIdx.y > M.g.N) return;
    const int ns = (M.g.I + kRomsCols - 1) / kRomsCols, by = mb.y / ns, bx = mb.y - by * ns;
    const long o3 = M.off3;
    roms_rhs3d_rows(M.g, u + o3, v + o3, Hu + o3, Hv + o3, Hz + M.offN, ru + o3, rv + o3, bx * kRomsCols,
                    (by * kRomsWarps + (int)(threadIdx.x >> 5)) * nrows, nrows, (int)blockIdx.y);
}
template <typename R>
__global__ void __launch_bounds__(128) k_roms_rhs3d_point(Geo<R> g, const R *u, const R *v, const R *Hu, const R *Hv,
                                                          const R *Hz, R *ru, R *rv) {
    roms_rhs3d_point(g, u, v, Hu, Hv, Hz, ru, rv, tid_flat(), (int)blockIdx.y, (int)gridDim.y);
}
template <typename R>
__global__ void __launch_bounds__(128) kb_roms_rhs3d_point(const Member<R> *mt, const int2 *bm, const R *u, const R *v,
                                                           const R *Hu, const R *Hv, const R *Hz, R *ru, R *rv) {
    const MemberAt<R> m = member_at(mt, bm, 128);
    roms_rhs3d_point(m.g, u + m.o3, v + m.o3, Hu + m.o3, Hv + m.o3, Hz + m.oN, ru + m.o3, rv + m.o3, m.p, (int)blockIdx.y,
                     (int)gridDim.y);
}
template <typename R>
__global__ void __launch_bounds__(256) k_roms_stress3d(Geo<R> g, const R *u, const R *v, R *ru,
                                                       R *rv, const R *sustr, const R *svstr,
                                                       R rdrag2) {
    roms_stress3d_at(g, u, v, ru, rv, sustr, svstr, rdrag2, tid_flat());
}
template <typename R>
__global__ void __launch_bounds__(256) kb_roms_stress3d(const Member<R> *mt, const int2 *bm,
                                                        const R *u, const R *v, R *ru, R *rv,
                                                        const R *sustr, const R *svstr,
                                                        R rdrag2) {
    const MemberAt<R> m = member_at(mt, bm, 256);
    roms_stress3d_at(m.g, u + m.o3, v + m.o3, ru + m.o3, rv + m.o3, sustr + m.o2, svstr + m.o2,
                     rdrag2, m.p);
}
// A point block's U columns and its V columns are consecutive blocks: Hz, Akv, z_r and W are then read
// from DRAM once for both.
template <typename R, typename Off, bool SHORT>
__global__ void __launch_bounds__(roms_col_threads<R>(), roms_col_blocks<R>(SHORT)) k_roms_step3d(
    Geo<R> g, R *u, R *v, RomsRhs<R> ru, RomsRhs<R> rv, R c0, R c1, R c2, R *ubar_n, R *vbar_n, R *ubar_s,
    R *vbar_s, const R *Hz, const R *Akv, const R *z_r, const R *W, const double *DU, const double *DV, R dt,
    R lamdt) {
    constexpr int T = roms_col_threads<R>();
    extern __shared__ __align__(16) unsigned char col_smem[];
    roms_step3d_at<R, T, Off, SHORT>(g, u, v, ru, rv, c0, c1, c2, ubar_n, vbar_n, ubar_s, vbar_s, Hz, Akv, z_r, W, DU, DV,
                         dt, lamdt, (long)(blockIdx.x >> 1) * T + threadIdx.x, blockIdx.x & 1,
                         reinterpret_cast<R *>(col_smem) + threadIdx.x);
}
template <typename R, typename Off, bool SHORT>
__global__ void __launch_bounds__(roms_col_threads<R>(), roms_col_blocks<R>(SHORT)) kb_roms_step3d(
    const Member<R> *mt, const int2 *bm, R *u, R *v, RomsRhs<R> ru, RomsRhs<R> rv, R c0, R c1, R c2, R *ubar_n,
    R *vbar_n, R *ubar_s, R *vbar_s, const R *Hz, const R *Akv, const R *z_r, const R *W, const double *DU,
    const double *DV, R dt, R lamdt) {
    constexpr int T = roms_col_threads<R>(), kPart = 128 / T;   // blocks of T columns in a block of the map
    extern __shared__ __align__(16) unsigned char col_smem[];
    const int2 mb = bm[blockIdx.x / (2 * kPart)];
    const Member<R> &M = mt[mb.x];
    const int part = (int)(blockIdx.x >> 1) % kPart;
    const long o3 = M.off3, o2 = M.off2;
    const RomsRhs<R> a{ru.r0 + o3, ru.r1 + o3, ru.r2 + o3}, b{rv.r0 + o3, rv.r1 + o3, rv.r2 + o3};
    roms_step3d_at<R, T, Off, SHORT>(M.g, u + o3, v + o3, a, b, c0, c1, c2, ubar_n + o2, vbar_n + o2, ubar_s + o2,
                         vbar_s + o2, Hz + M.offN, Akv + o3, z_r + M.offN, W + o3, DU + o2, DV + o2, dt, lamdt,
                         (long)mb.y * 128 + part * T + threadIdx.x, blockIdx.x & 1,
                         reinterpret_cast<R *>(col_smem) + threadIdx.x);
}
template <typename R>
__global__ void __launch_bounds__(256) k_roms_walls3d(Geo<R> g, R *u, R *v) {
    roms_walls3d_at(g, u, v, tid_flat());
}
template <typename R>
__global__ void __launch_bounds__(256) kb_roms_walls3d(const Member<R> *mt, const int2 *bm, R *u,
                                                       R *v) {
    const MemberAt<R> m = member_at(mt, bm, 256);
    roms_walls3d_at(m.g, u + m.o3, v + m.o3, m.p);
}

constexpr int kGridY = 65535;   // blocks a grid holds along y
// Rows a warp walks: at least as many as a grid of kRomsWarps warps a block needs for J rows.
inline int roms_fit_rows(int rows, int J) {
    const int least = (int)(((long)J + (long)kGridY * kRomsWarps - 1) / ((long)kGridY * kRomsWarps));
    return rows > least ? rows : least;
}

template <typename R>
cudaError_t Ops<R>::roms_phase(const sf_ctx *c, const RomsArgs<R> &a, cudaStream_t s) {
    const int B = 32 * kRomsWarps;
    if (a.phase == 3) {
        const int ny = (c->J + kSubRows - 4) / (kSubRows - 3);
        dim3 grid((c->I + kSubCols - 1) / kSubCols, ny < kGridY ? ny : kGridY, (ny + kGridY - 1) / kGridY);
        if (c->nmem > 1) grid = dim3(c->nbm_sub);
        // few tiles: one node's latency counts, everything in registers (514 x 258 nodes, 580 tiles, FP32:
        // 367 us a loop of 52 substeps against 437; 130 x 66, FP64: 220 against 229); many: blocks per
        // SM count (642 x 322, 864 tiles, FP32: 480 against 512; 514 x 258, FP64: 638 against 716; at
        // 258 x 130, 150 tiles, FP64 takes 333 and 336)
        return (long)grid.x * grid.y * grid.z >= (sizeof(R) == 4 ? 720 : 200) ? roms_sub_launch<R, true>(c, a, grid, s)
                                                                              : roms_sub_launch<R, false>(c, a, grid, s);
    }
    if (a.phase != 2 && !roms_by_strips(c)) {
        for (int mom = 0; mom < 2; ++mom) {
            cudaError_t e;
            if (c->nmem > 1) {
                auto k = a.phase == 0 ? (mom ? kb_roms_point<R, 0, true> : kb_roms_point<R, 0, false>)
                                      : (mom ? kb_roms_point<R, 1, true> : kb_roms_point<R, 1, false>);
                e = launch_dep(c, k, c->nbm_pt, 256, 0, s, mt<R>(c), c->bm_pt, a);
            } else {
                auto k = a.phase == 0 ? (mom ? k_roms_point<R, 0, true> : k_roms_point<R, 0, false>)
                                      : (mom ? k_roms_point<R, 1, true> : k_roms_point<R, 1, false>);
                e = launch_dep(c, k, blocks_for(c->s2, 256), 256, 0, s, geo(c), a);
            }
            if (e != cudaSuccess) return e;
        }
        return cudaSuccess;
    }
    if (c->nmem > 1) {
        if (a.phase == 2)
            return launch_dep(c, kb_roms_acc<R>, c->nbm_pt, 256, 0, s, mt<R>(c), c->bm_pt, a);
        auto k = a.phase == 0 ? kb_roms_phase<R, 0> : kb_roms_phase<R, 1>;
        return launch_dep(c, k, c->nbm_roms, B, 0, s, mt<R>(c), c->bm_roms, a, c->roms_rows);
    }
    if (a.phase == 2) return launch_dep(c, k_roms_acc<R>, blocks_for(c->s2, 256), 256, 0, s, geo(c), a);
    const int rows = roms_fit_rows(c->roms_rows, c->J);
    const dim3 grid((c->I + kRomsCols - 1) / kRomsCols, (c->J + rows * kRomsWarps - 1) / (rows * kRomsWarps));
    auto k = a.phase == 0 ? k_roms_phase<R, 0> : k_roms_phase<R, 1>;
    return launch_dep(c, k, grid, B, 0, s, geo(c), a, rows);
}
template <typename R>
cudaError_t Ops<R>::roms_stress3d(const sf_ctx *c, const R *u, const R *v, R *ru, R *rv,
                                  const R *sustr, const R *svstr, double rdrag2, cudaStream_t s) {
    if (c->nmem > 1)
        kb_roms_stress3d<R><<<c->nbm_pt, 256, 0, s>>>(mt<R>(c), c->bm_pt, u, v, ru, rv, sustr,
                                                      svstr, (R)rdrag2);
    else
        k_roms_stress3d<R><<<blocks_for(c->s2, 256), 256, 0, s>>>(geo(c), u, v, ru, rv, sustr,
                                                                    svstr, (R)rdrag2);
    return cudaGetLastError();
}
template <typename R>
cudaError_t Ops<R>::roms_rhs3d(const sf_ctx *c, const R *u, const R *v, const R *Huon,
                               const R *Hvom, const R *Hz, R *ru, R *rv, cudaStream_t s) {
    const int B = 32 * kRomsWarps;
    // Strips where enough of their 29 columns exist.  us by points and by strips, 30 levels, FP32: 14 x 14285 points
    // 63 and 67, 17 x 11764 62 and 58, 20 x 10000 62 and 52; 5 levels: 17 x 58823 48 and 50, 20 x 50000 48 and 46; FP64,
    // 30 levels: 12 x 16666 108 and 112, 14 x 14285 108 and 100.  Ensembles, whose strips have the phases' fewer rows,
    // 32 levels: 22 columns (40 of 66 x 34) FP32 28 and 39, FP64 53 and 58; 27 (12 of 300 x 140) 152 and 129, 228 and 200.
    const int N = c->nmem > 1 ? c->maxN : c->N;
    const int least = c->nmem > 1 ? 24 : (sizeof(R) == 8 ? 14 : (N < 10 ? 19 : 15));
    if (c->s2 < least * c->roms_strip_rows) {
        // by points: the levels of a point over as many threads as small basins need (5 x 6000 points of 30 levels, FP32,
        // all, 2, 1: 12, 15, 25 us; 5 x 40000 65, 62, 79; 4 members of 8 x 2000, 32 levels, all, 4, 2, 1: 24, 20, 20, 28)
        const int levels = c->s2 < (1L << 15) ? N + 1 : c->s2 < (1L << 18) ? 4 : 2;
        if (c->nmem > 1)
            kb_roms_rhs3d_point<R><<<dim3(c->nbm_128, levels), 128, 0, s>>>(mt<R>(c), c->bm_128, u, v, Huon, Hvom, Hz, ru, rv);
        else
            k_roms_rhs3d_point<R><<<dim3(blocks_for(c->s2, 128), levels), 128, 0, s>>>(geo(c), u, v, Huon, Hvom, Hz, ru, rv);
    } else if (c->nmem > 1) {
        kb_roms_rhs3d<R><<<dim3(c->nbm_roms, c->maxN + 1), B, 0, s>>>(mt<R>(c), c->bm_roms, u, v, Huon, Hvom, Hz, ru,
                                                                     rv, c->roms_rows);
    } else {
        // rows a warp walks: 8 (1026 x 514 x 50 in FP32: 4, 8, 16, 32, 64 rows 0.177, 0.158, 0.162, 0.168,
        // 0.184 ms), 32 on large grids (2050 x 1026 x 50: 0.685, 0.618, 0.627, 0.605, 0.584)
        const int rows = roms_fit_rows(c->s2 >= (1L << 20) ? 32 : 8, c->J);
        const dim3 grid((c->I + kRomsCols - 1) / kRomsCols, (c->J + rows * kRomsWarps - 1) / (rows * kRomsWarps),
                        c->N + 1);
        k_roms_rhs3d<R><<<grid, B, 0, s>>>(geo(c), u, v, Huon, Hvom, Hz, ru, rv, rows);
    }
    return cudaGetLastError();
}
template <typename R>
cudaError_t Ops<R>::roms_step3d(const sf_ctx *c, R *u, R *v, const R *const *ru, const R *const *rv,
                                const double *coef, R *ubar_n, R *vbar_n, R *ubar_s, R *vbar_s,
                                const R *Hz, const R *Akv, const R *z_r, const R *W,
                                const double *DU, const double *DV, double dt, double lamdt,
                                cudaStream_t s) {
    const RomsRhs<R> a{ru[0], ru[1], ru[2]}, b{rv[0], rv[1], rv[2]};
    constexpr int T = roms_col_threads<R>();
    static bool done[64] = {};   // the raised shared-memory limit, once on each device
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= 64 || !done[dev]) {
        const auto at = cudaFuncAttributeMaxDynamicSharedMemorySize;
        const int most = 2 * kRomsMaxN * T * (int)sizeof(R);
        for (auto k : {k_roms_step3d<R, int, false>, k_roms_step3d<R, long, false>})
            if (e == cudaSuccess) e = cudaFuncSetAttribute(k, at, most);
        for (auto k : {kb_roms_step3d<R, int, false>, kb_roms_step3d<R, long, false>})
            if (e == cudaSuccess) e = cudaFuncSetAttribute(k, at, most);
        if (e != cudaSuccess) return e;
        if (dev >= 0 && dev < 64) done[dev] = true;
    }
    const int N = c->nmem > 1 ? c->maxN : c->N, smem = 2 * N * T * (int)sizeof(R);
    // 32-bit offsets within a member's field: (N + 2) levels of at most the pool's points
    const bool fits = (long)(N + 2) * c->s2 < (1L << 31);
    const bool brief = fits && N <= kRomsShortN;   // at most 16 KB of shared memory a block
    if (c->nmem > 1)
        (brief ? kb_roms_step3d<R, int, true>
         : fits ? kb_roms_step3d<R, int, false> : kb_roms_step3d<R, long, false>)<<<2 * (128 / T) * c->nbm_128, T, smem, s>>>(
            mt<R>(c), c->bm_128, u, v, a, b, (R)coef[0], (R)coef[1], (R)coef[2], ubar_n, vbar_n, ubar_s, vbar_s,
            Hz, Akv, z_r, W, DU, DV, (R)dt, (R)lamdt);
    else
        (brief ? k_roms_step3d<R, int, true>
         : fits ? k_roms_step3d<R, int, false> : k_roms_step3d<R, long, false>)<<<2 * blocks_for(c->s2, T), T, smem, s>>>(
            geo(c), u, v, a, b, (R)coef[0], (R)coef[1], (R)coef[2], ubar_n, vbar_n, ubar_s, vbar_s, Hz, Akv, z_r,
            W, DU, DV, (R)dt, (R)lamdt);
    return cudaGetLastError();
}
template <typename R>
cudaError_t Ops<R>::roms_walls3d(const sf_ctx *c, R *u, R *v, cudaStream_t s) {
    if (c->nmem > 1)
        kb_roms_walls3d<R><<<c->nbm_pt, 256, 0, s>>>(mt<R>(c), c->bm_pt, u, v);
    else
        k_roms_walls3d<R><<<blocks_for(c->s2, 256), 256, 0, s>>>(geo(c), u, v);
    return cudaGetLastError();
}

}  // namespace sf
