// gft_shared_body.cuh -- the site update of the tiled kernels with every loop and
// every transported doublet computed once per tile.
//
// A site's lower loops are its back neighbours' upper loops, turned by its own links
// (gft_step_body.cuh), and its backward transports are theirs forward.  In an x-march
// the x neighbour's come from the thread's own last site (XCarry); here the y and z
// neighbours' come from their threads.  The update is cut in two:
//   site_open  : upper loops, forward and backward transports with the plane x + 1 --
//                everything a site computes from itself and its forward neighbours;
//   site_close : what the back neighbours hand over (Handed), the past level, the
//                leapfrog and the stores -- own-site values only.
// The y neighbour's values pass through shared memory under the plane's one CTA
// barrier, which lies between the two; the z neighbour's by warp shuffle.  The row
// y0 - 1 and the column z0 - 1 belong to other tiles: their values for this tile are
// computed by TY + TZ lanes of two of the tile's warps, a different pair each plane
// (halo_hand_over).
//
// The mixed form's tiled steps are bound by instruction issue (66 to 74 % of the slots, 16 warps per
// SM); the FP64 ones wait on chains of FP64 operations with 8 warps per SM (issue 36 to 39 %, FP64
// pipe 48 %).  Per site the lower loops fall from four (two carried) to none, their sines and the two
// backward transports with their sines and cosines too; three turns remain: 1,306 warp instructions
// per 32 sites at SM 128^3, the halo row and column (4 % of the work of an 8 x 32 tile) included.  us
// per step, against every thread computing its own lower loops (site_step with CARRY): SM mixed 256^3
// 896 -> 831, 128^3 140 -> 134, logging 256^3 1147 -> 1110; FP64 2HDM 192^3 1090 -> 1076, logging 1600 ->
// 1617 (one thread per site 1233, 1996); FP64 SM 256^3 1793 -> 1854, logging 2993 -> 2985: there the
// sines saved no longer pay.  The float 2HDM's tiles keep site_step (hands_over).
#pragma once

#include "gft_step_body.cuh"

namespace gft {

// What a site hands to its +e_d neighbour (d = 1, 2; a < b the other two directions): the
// vector parts of link d's upper loops in the planes with a and b, the sines of F_ad and
// F_bd, and the doublets transported along link d.  2 + ND quads.
template <class C, int ND>
struct Handed {
    C fa[3], sa;
    C fb[3], sb;
    Q<C> t[ND];
};

// A site between its two halves.  r[i]: the sum over planes of weight times the vector
// that link i's lower loops are, before the turn by U_i.
template <class C, int ND>
struct OpenSite {
    Q<C> U[3], fc[ND], D[ND];
    C th[3], Mg[3][3], r[3][3], MgY[3];
    C mag_e, plaq2, plaq1, grad_e;
    double pot_e;
};

// Adds what the back neighbour of direction d handed over, weight l = dt^2 / dx_d^2.
template <class C, int ND>
__device__ __forceinline__ void receive(OpenSite<C, ND>& o, int a, int b, C l, const Handed<C, ND>& h)
{
#pragma unroll
    for (int k = 0; k < 3; k++) {
        o.r[a][k] += l * h.fa[k];
        o.r[b][k] += l * h.fb[k];
    }
    o.MgY[a] += l * h.sa;
    o.MgY[b] += l * h.sb;
#pragma unroll
    for (int db = 0; db < ND; db++) o.D[db] = qadd_scaled(o.D[db], l, h.t[db]);
}

template <class S, int MODEL, bool ENERGY, class A, class R, int ND>
__device__ __forceinline__ void site_open(const StepParams& P, const KConst<S>& F, const A& acc, const Stencil<R>& n,
                                          XCarry<S, ND>& carry, OpenSite<S, ND>& o, Handed<S, ND>& hy,
                                          Handed<S, ND>& hz)
{
    using C = S;
    const C l[3] = {F.ldt[0], F.ldt[1], F.ldt[2]};
#pragma unroll
    for (int a = 0; a < 3; a++) {
        o.U[a] = acc.q(a, n.c);
        o.th[a] = acc.th(a, n.c);
    }

    // ---- own-site terms and what the x neighbour handed over ----
#pragma unroll
    for (int db = 0; db < ND; db++) o.fc[db] = acc.ph(db, n.c);
    o.pot_e = site_potential<MODEL, ENERGY>(P, F, o.fc, o.D);
#pragma unroll
    for (int db = 0; db < ND; db++) o.D[db] = qadd_scaled(o.D[db], l[0], carry.t0[db]);
    o.MgY[0] = (C)0;
    o.MgY[1] = -l[0] * carry.s01;
    o.MgY[2] = -l[0] * carry.s02;
#pragma unroll
    for (int k = 0; k < 3; k++) {
        o.r[0][k] = (C)0;
        o.r[1][k] = l[0] * carry.v01[k];
        o.r[2][k] = l[0] * carry.v02[k];
#pragma unroll
        for (int i = 0; i < 3; i++) o.Mg[i][k] = (C)0;
    }
    if (ENERGY) o.mag_e = o.plaq2 = o.plaq1 = o.grad_e = (C)0;

    // ---- upper loops ----
#pragma unroll
    for (int pl = 0; pl < 3; pl++) {
        const int i = (pl == 2) ? 1 : 0;
        const int j = (pl == 0) ? 1 : 2;
        const C Fa = o.th[i] + acc.th(j, n.p[i]) - acc.th(i, n.p[j]) - o.th[j];  // F_ij
        const C sF = gsin(Fa);
        o.MgY[i] -= sF * l[j];
        o.MgY[j] += sF * l[i];
        C vi[3], vj[3];  // the forces on links i and j are vi and -vj
        const C w = plaq_forces(acc.q(j, n.p[i]), acc.q(i, n.p[j]), o.U[i], o.U[j], vi, vj);
#pragma unroll
        for (int k = 0; k < 3; k++) {
            o.Mg[i][k] += l[j] * vi[k];
            o.Mg[j][k] -= l[i] * vj[k];
            if (pl == 0) {
                carry.v01[k] = vi[k];
                hy.fa[k] = -vj[k];
            } else if (pl == 1) {
                carry.v02[k] = vi[k];
                hz.fa[k] = -vj[k];
            } else {
                hy.fb[k] = vi[k];
                hz.fb[k] = -vj[k];
            }
        }
        if (pl == 0) carry.s01 = hy.sa = sF;
        if (pl == 1) carry.s02 = hz.sa = sF;
        if (pl == 2) {
            hy.sb = -sF;
            hz.sb = sF;
        }
        if (ENERGY) {
            const C hF = gsin((C)0.5 * Fa), omc = (C)2 * hF * hF;  // 1 - cos F
            const C omt = one_minus_trace(Q<C>{w, vi[0], vi[1], vi[2]});
            o.mag_e += F.e_plaq[pl] * (F.inv_g_sqr * omt + F.inv_gp_sqr * omc);
            o.plaq2 += (C)1 - omt;
            o.plaq1 += (C)1 - omc;
        }
    }

    // ---- transports and currents (four times the reference's; the 1/4 is in cY and cI) ----
#pragma unroll
    for (int a = 0; a < 3; a++) {
        C sn, cs;
        gsincos(o.th[a], sn, cs);
#pragma unroll
        for (int db = 0; db < ND; db++) {
            const Q<C> g = acc.ph(db, n.p[a]);
            o.D[db] = qadd_scaled(o.D[db], l[a], transport_back(o.U[a], cs, sn, g));
            const Q<C> u = transport(o.U[a], cs, sn, o.fc[db]);
            const C up = u.w * g.x - u.x * g.w, lo = u.y * g.z - u.z * g.y;
            o.MgY[a] += F.cY * (up + lo);
            o.Mg[a][0] += F.cI * (u.w * g.z - u.x * g.y + u.y * g.x - u.z * g.w);
            o.Mg[a][1] += F.cI * (-u.w * g.y - u.x * g.z + u.y * g.w + u.z * g.x);
            o.Mg[a][2] += F.cI * (up - lo);
            if (ENERGY) {
                const C e0 = g.w - u.w, e1 = g.x - u.x, e2 = g.y - u.y, e3 = g.z - u.z;
                o.grad_e += F.e_grad[a] * (e0 * e0 + e1 * e1 + e2 * e2 + e3 * e3);
            }
            if (a == 0) carry.t0[db] = u;
            if (a == 1) hy.t[db] = u;
            if (a == 2) hz.t[db] = u;
        }
    }
}

// What the site c of a staged plane hands to its +e_d neighbour, d (1 or 2)
// a run-time value of the lane; p0, p1, p2: the cells of x + e_a.
template <class S, class A, class R, int ND>
__device__ __forceinline__ void halo_hand_over(const A& acc, int d, R c, R p0, R p1, R p2, Handed<S, ND>& h)
{
    using C = S;
    const int b = 3 - d;
    const R pd = (d == 1) ? p1 : p2, pb = (d == 1) ? p2 : p1;
    const Q<C> Ud = acc.q(d, c);
    const C thd = acc.th(d, c);
    C vj[3];
    // link d's loop in plane o from C = U_o(x+d)^dag U_d(x+o) and D = U_o U_d^dag
    plaq_forces(acc.q(0, pd), acc.q(d, p0), Ud, acc.q(0, c), h.fa, vj);
    plaq_forces(acc.q(b, pd), acc.q(d, pb), Ud, acc.q(b, c), h.fb, vj);
    h.sa = gsin(acc.th(0, c) + acc.th(d, p0) - acc.th(0, pd) - thd);
    h.sb = gsin(acc.th(b, c) + acc.th(d, pb) - acc.th(b, pd) - thd);
    C sn, cs;
    gsincos(thd, sn, cs);
#pragma unroll
    for (int db = 0; db < ND; db++) h.t[db] = transport(Ud, cs, sn, acc.ph(db, c));
}

template <class S, bool ENERGY, int ND, class PV>
__device__ __forceinline__ void site_close(const StepParams& P, const KConst<S>& F, OpenSite<S, ND>& o, const PV& past,
                                           double (&obs)[kObsCount], unsigned& warn, bool count)
{
    using C = S;
    const unsigned warn_in = warn;
#pragma unroll
    for (int i = 0; i < 3; i++) add_turned(o.Mg[i], (C)1, o.U[i], o.r[i]);
    C kin_e = (C)0, phisq = (C)0, elec_e = (C)0, check = (C)0;
#pragma unroll
    for (int db = 0; db < ND; db++)
        leapfrog_doublet<ENERGY>(F, o.fc[db], past.ph(db), o.D[db], past.at.L.ph[db], past.at.s, kin_e, phisq, check);
    leapfrog_links<ENERGY>(F, o.U, o.th, o.Mg, o.MgY, past, elec_e, warn, check);
    if (!isfinite(check)) warn |= kWarnNonFinite;
    if (!count) {
        warn = warn_in;
        return;
    }
    if (ENERGY)
        record_energies(P, past.at.s, o.pot_e, o.grad_e, kin_e, o.mag_e, elec_e, o.plaq2, o.plaq1, phisq, obs);
}

}  // namespace gft
