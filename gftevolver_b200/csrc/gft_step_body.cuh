// gft_step_body.cuh -- the per-site leapfrog update of the throughput forms,
// written once against a field accessor so that the same arithmetic serves the
// global-memory kernel (neighbours read through L1/L2) and the tiled kernel
// (neighbours read from TMA-staged shared-memory planes).
//
// Physics: the reference's per-site update (Core/Source/Model.cpp:339-373,
// WilsonLoops/Source/StandardModel.cpp:324-514, Gradients/Source/StandardModel.cpp:72-100,
// 272-363, Potentials/Source/SO_N.cpp:57-75, Potentials/Source/Double_SO_N.cpp:244-341),
// reassociated:
//   * the reference builds, for every link i and plane j, the loops
//       P1 = U_j(x+i)^dag U_i(x+j) U_j(x) U_i(x)^dag,
//       P2 = U_i(x) U_j(x-j) U_i(x-j)^dag U_j(x+i-j)^dag,
//     renormalising intermediate products.  Here the upper loops of both links of a
//     plane come from two products (plaq_forces); the lower ones are summed as
//       SB_i = sum_j w_j U_j(x-j) U_i(x-j)^dag U_j(x+i-j)^dag
//     before the product with U_i (the vector part is linear), and in an x-march those
//     of the planes with x are the x-1 site's upper loops, turned:
//       P2 of link i in plane x = U_i(x) (P1 of link 0 at x-e_0 in plane i)^dag U_i(x)^dag.
//     Intermediate renormalisation is dropped: it changes products of unit quaternions
//     only at the rounding level.
//   * the U(1) plaquette angle of plane (i,j) is computed once for both links.
//   * sin, cos and asin are the range-reduced series of gft_math.cuh.
// Precision of the mixed form (C = float): operations that would lose
// precision in float are rearranged rather than widened -- the link momentum
// is vec((U_now - U_past) U_past^dag) (exactly vec(U_now U_past^dag) without
// the O(1) terms that cancel), leapfrog sums add a small increment to the
// current value with one rounding, and the renormalisation evaluates
// |U|^2 - 1 with fused multiply-adds.  Energies accumulate in FP64.
#pragma once

#include "gft_device.cuh"
#include "gft_math.cuh"

namespace gft {

__device__ __forceinline__ float sqrt_(float x) { return sqrtf(x); }
__device__ __forceinline__ double sqrt_(double x) { return sqrt(x); }

// Doublet phi rotated by the hypercharge phase (cos, sin) then acted on by the
// SU(2) quaternion u as the real 4x4 of Gradients/Source/StandardModel.cpp:94-97.
template <class C>
__device__ __forceinline__ Q<C> transport(Q<C> u, C cs, C sn, Q<C> f)
{
    const C h0 = cs * f.w - sn * f.x;
    const C h1 = cs * f.x + sn * f.w;
    const C h2 = cs * f.y - sn * f.z;
    const C h3 = cs * f.z + sn * f.y;
    Q<C> t;
    t.w = u.w * h0 - u.z * h1 + u.y * h2 - u.x * h3;
    t.x = u.z * h0 + u.w * h1 + u.x * h2 + u.y * h3;
    t.y = -u.y * h0 - u.x * h1 + u.w * h2 + u.z * h3;
    t.z = u.x * h0 - u.y * h1 - u.z * h2 + u.w * h3;
    return t;
}

// The inverse transport: acted on by the conjugate link, phase rotated back.
template <class C>
__device__ __forceinline__ Q<C> transport_back(Q<C> u, C cs, C sn, Q<C> f)
{
    return transport(qconj(u), cs, -sn, f);
}

// The isospin action alone (the 4x4 above on an already phase-rotated h); the
// Higgs-family SU(2) acts with the same matrix on (doublet-1, doublet-2)
// component pairs (Gradients/Source/TwoHDM.cpp:134-146).
template <class C>
__device__ __forceinline__ Q<C> su2_act(Q<C> u, Q<C> h)
{
    Q<C> t;
    t.w = u.w * h.w - u.z * h.x + u.y * h.y - u.x * h.z;
    t.x = u.z * h.w + u.w * h.x + u.x * h.y + u.y * h.z;
    t.y = -u.y * h.w - u.x * h.x + u.w * h.y + u.z * h.z;
    t.z = u.x * h.w - u.y * h.x - u.z * h.y + u.w * h.z;
    return t;
}

// Phase rotation of both complex pairs of a doublet by (cos, sin).
template <class C>
__device__ __forceinline__ Q<C> rot2(Q<C> f, C cs, C sn)
{
    return {cs * f.w - sn * f.x, cs * f.x + sn * f.w, cs * f.y - sn * f.z, cs * f.z + sn * f.y};
}

// Higgs-family part of the 2HDM transport (Gradients/Source/TwoHDM.cpp:118-146),
// applied to the two SM-transported doublets: U(1) = phase +theta_H on doublet 1
// and -theta_H on doublet 2 ((hc, hs) = cos, sin of theta_H, hs negated for the
// conjugate link); SU(2) = hu acting on (doublet 1, doublet 2) pairs.
template <int HF, class C>
__device__ __forceinline__ void hf_act(Q<C>& t1, Q<C>& t2, C hc, C hs, Q<C> hu)
{
    if constexpr (HF == kHfU1) {
        t1 = rot2(t1, hc, hs);
        t2 = rot2(t2, hc, -hs);
    } else if constexpr (HF == kHfSU2) {
        const Q<C> lo = su2_act(hu, Q<C>{t1.w, t1.x, t2.w, t2.x});
        const Q<C> hi = su2_act(hu, Q<C>{t1.y, t1.z, t2.y, t2.z});
        t1 = {lo.w, lo.x, hi.w, hi.x};
        t2 = {lo.y, lo.z, hi.y, hi.z};
    }
}

// Leapfrog update of a site's three SU(2) links from the vector parts R[d] of
// u = U(t+dt) U(t)^dag (WilsonLoops/Source/StandardModel.cpp:478-504), stored to
// out[d][s] and added to `check`.  U(t+dt) = normalise(u U(t)) is written as U + correction:
// u = (sqrt(1 - |R|^2), R) is a unit quaternion, so |u U|^2 - 1 = |U|^2 - 1 =: e, and with
// f = 1/sqrt(1+e) - 1 = -e/2 + 3e^2/8
//   U(t+dt) = U + (u0 - 1 + f u0, (1 + f) R) U,
// one rounding at the end.  f R counts for links that are not unit to the working precision
// (float words in the FP64 form, say): without it the new link keeps e |R|^2 / 2 of their norm.
// Its four multiply-adds per link cost 2 to 3 % (SM mixed 128^3, 40 steps: 5733 -> 5887 us; 2HDM
// FP64 192^3, 10 steps: 12732 -> 13339), and a branch that only such links take costs the same.
// The series of u0 - 1 serves where all three |R|^2 are small; one test for the three.
template <class C, class S>
__device__ __forceinline__ void su2_advance3(const Q<C> (&U)[3], const C (&R)[3][3], S* const (&out)[3], int s,
                                             unsigned& warn, C& check)
{
    C cm[3], u0m1[3];
#pragma unroll
    for (int d = 0; d < 3; d++) cm[d] = R[d][0] * R[d][0] + R[d][1] * R[d][1] + R[d][2] * R[d][2];
    MaxAbs<C> m;
#pragma unroll
    for (int d = 0; d < 3; d++) m.add(cm[d]);
    if (m.exceeds(Sqrt1mSeries<C>::limit)) {
#pragma unroll
        for (int d = 0; d < 3; d++) {
            if (cm[d] > (C)1) warn |= kWarnSqrt;
            u0m1[d] = sqrt1m_minus1(cm[d]);
        }
    } else {
#pragma unroll
        for (int d = 0; d < 3; d++) u0m1[d] = sqrt1m_series(cm[d]);
    }
#pragma unroll
    for (int d = 0; d < 3; d++) {
        const Q<C> Un = U[d];
        C e = fma(Un.w, Un.w, (C)-1);
        e = fma(Un.x, Un.x, e);
        e = fma(Un.y, Un.y, e);
        e = fma(Un.z, Un.z, e);
        const C f = e * ((C)0.375 * e - (C)0.5), a = fma(f, u0m1[d], u0m1[d] + f);
        const Q<C> dU = qmul(Q<C>{a, fma(f, R[d][0], R[d][0]), fma(f, R[d][1], R[d][1]), fma(f, R[d][2], R[d][2])}, Un);
        check += a;  // non-finite if a word of U or R is
        st4(out[d], s, Un.w + dU.w, Un.x + dU.x, Un.y + dU.y, Un.z + dU.z);
    }
}

// 1 - a0/|a| in the compute type without cancellation: |vec a|^2 / (|a| (|a| + a0))
// when a0 >= 0, else 1 - a0/|a| directly (no cancellation there either).
template <class C>
__device__ __forceinline__ C one_minus_trace(Q<C> a)
{
    const C v2 = a.x * a.x + a.y * a.y + a.z * a.z;
    const C nrm = sqrt_(a.w * a.w + v2);
    return (a.w >= (C)0) ? v2 / (nrm * (nrm + a.w)) : (C)1 - a.w / nrm;
}
// The mixed form's energy terms: the same expression with the square root and the
// division by Newton-refined hardware approximations (one_minus_cos_nr), a fifth
// of the instructions of the IEEE operations; the FP64 forms keep those.
template <>
__device__ __forceinline__ float one_minus_trace<float>(Q<float> a)
{
    return one_minus_cos_nr(a.w, a.x * a.x + a.y * a.y + a.z * a.z);
}

// Neighbour references of one site, in the accessor's own reference type:
//   c = x, m[a] = x - e_a, p[a] = x + e_a, dg(i, j) = x + e_i - e_j (i != j).
template <class R>
struct Stencil {
    R c, m[3], p[3];
    R d01, d02, d10, d12, d20, d21;
    __device__ __forceinline__ R dg(int i, int j) const
    {
        return (i == 0) ? (j == 1 ? d01 : d02) : (i == 1) ? (j == 0 ? d10 : d12) : (j == 0 ? d20 : d21);
    }
};

// Values a site computes that its +x neighbour needs, carried along an x-march:
// the sines of the (0,1) and (0,2) plaquette angles, which are the x+e_0
// site's lower U(1) loop angles; the vector parts of the x link's (0,1) and (0,2)
// plaquettes, which turned by U_1 and U_2 are the x+e_0 site's lower loops of the
// links 1 and 2; and the doublet transported along the x link, U_0(x) R(theta_0(x))
// phi(x), which is the x+e_0 site's D- term.  With them a site reads nothing of
// the plane x - 1.
template <class C, int ND>
struct XCarry {
    C s01, s02;
    C v01[3], v02[3];
    Q<C> t0[ND];
};

// Own-site past level (read, then overwritten with t + dt).  LV is LevelPtrs<S>, or any
// struct with its q / th / ph members when no Higgs-family field is evolved.
template <class S, class LV = LevelPtrs<S>>
struct PastSite {
    LV L;
    int s;
};

// Its values: EARLY, loaded together by load() so that their latency overlaps arithmetic
// (plain steps); else each where it is used (logging steps have no registers to spare).
template <class S, int ND, class LV, bool EARLY>
struct PastValues {
    PastSite<S, LV> at;
    Q<S> f[ND], u[3];
    S t[3];
    __device__ __forceinline__ void load()
    {
        if (!EARLY) return;
#pragma unroll
        for (int db = 0; db < ND; db++) f[db] = ld4<S>(at.L.ph[db], at.s);
#pragma unroll
        for (int d = 0; d < 3; d++) {
            u[d] = ld4<S>(at.L.q[d], at.s);
            t[d] = ld1<S>(at.L.th[d], at.s);
        }
    }
    __device__ __forceinline__ Q<S> ph(int db) const { return EARLY ? f[db] : ld4<S>(at.L.ph[db], at.s); }
    __device__ __forceinline__ Q<S> q(int d) const { return EARLY ? u[d] : ld4<S>(at.L.q[d], at.s); }
    __device__ __forceinline__ S th(int d) const { return EARLY ? t[d] : ld1<S>(at.L.th[d], at.s); }
};

// A thread's total energy from its component sums, set once after its last site
// (no per-site accumulator held through the update).
__device__ __forceinline__ void energy_total(double (&obs)[kObsCount])
{
    obs[kObsEnergy] = obs[kObsPotential] + obs[kObsGradient] + obs[kObsKinetic] + obs[kObsMagnetic] + obs[kObsElectric];
}

// Both SU(2) plaquette forces of a plane (i, j) from its four links: with
// C = U_j(x+i)^dag U_i(x+j) and D = U_j(x) U_i(x)^dag the loop of link i is C D and
// that of link j is (D C)^dag, so the vector parts are vi = s - k and vj = s + k of
// s = c_0 d + d_0 c and k = c x d (the force on link j is -vj).  Returns the scalar
// part of C D (the plaquette trace; the same for both loops).
template <class C>
__device__ __forceinline__ C plaq_forces(Q<C> Uj_pi, Q<C> Ui_pj, Q<C> Ui, Q<C> Uj, C (&vi)[3], C (&vj)[3])
{
    const Q<C> c = qmul(qconj(Uj_pi), Ui_pj);
    const Q<C> d = qmul(Uj, qconj(Ui));
    const C s1 = c.w * d.x + d.w * c.x, s2 = c.w * d.y + d.w * c.y, s3 = c.w * d.z + d.w * c.z;
    const C k1 = c.y * d.z - c.z * d.y, k2 = c.z * d.x - c.x * d.z, k3 = c.x * d.y - c.y * d.x;
    vi[0] = s1 - k1;
    vi[1] = s2 - k2;
    vi[2] = s3 - k3;
    vj[0] = s1 + k1;
    vj[1] = s2 + k2;
    vj[2] = s3 + k3;
    return c.w * d.w - c.x * d.x - c.y * d.y - c.z * d.z;
}

// m += s vec(u v u^dag) for a unit quaternion u and a vector part v:
// u v u^dag = v + 2 (u x t - u_0 t) with t = u x v.
template <class C>
__device__ __forceinline__ void add_turned(C (&m)[3], C s, Q<C> u, const C (&v)[3])
{
    const C t1 = u.y * v[2] - u.z * v[1], t2 = u.z * v[0] - u.x * v[2], t3 = u.x * v[1] - u.y * v[0];
    const C r1 = u.y * t3 - u.z * t2 - u.w * t1;
    const C r2 = u.z * t1 - u.x * t3 - u.w * t2;
    const C r3 = u.x * t2 - u.y * t1 - u.w * t3;
    const C s2 = s + s;
    m[0] += s * v[0] + s2 * r1;
    m[1] += s * v[1] + s2 * r2;
    m[2] += s * v[2] + s2 * r3;
}

// The SU(2) magnetic force on the three links of a site, sum_j l_j (vec P1 - vec P2)
// (the loops at the head of this file), from link accessor q(d, R).  CARRY: the
// lower loops in the planes with x come from the x - 1 site's plaquettes w01, w02,
// which this site's replace.  trace(plane, scalar part, vector part) receives the
// upper plaquettes where the caller wants their energy.
template <bool CARRY, class C, class R, class QA, class Trace>
__device__ __forceinline__ void su2_force(QA&& q, const Stencil<R>& n, const Q<C> (&U)[3], const C (&l)[3], C (&w01)[3],
                                          C (&w02)[3], C (&Mg)[3][3], Trace&& trace)
{
#pragma unroll
    for (int i = 0; i < 3; i++) Mg[i][0] = Mg[i][1] = Mg[i][2] = (C)0;
    if constexpr (CARRY) {
        add_turned(Mg[1], l[0], U[1], w01);
        add_turned(Mg[2], l[0], U[2], w02);
    }
#pragma unroll
    for (int pl = 0; pl < 3; pl++) {
        const int i = (pl == 2) ? 1 : 0;
        const int j = (pl == 0) ? 1 : 2;
        C vi[3], vj[3];
        const C w = plaq_forces(q(j, n.p[i]), q(i, n.p[j]), U[i], U[j], vi, vj);
#pragma unroll
        for (int k = 0; k < 3; k++) {
            Mg[i][k] += l[j] * vi[k];
            Mg[j][k] -= l[i] * vj[k];
            if constexpr (CARRY) {
                if (pl == 0) w01[k] = vi[k];
                if (pl == 1) w02[k] = vi[k];
            }
        }
        trace(pl, Q<C>{w, vi[0], vi[1], vi[2]});
    }
#pragma unroll
    for (int i = 0; i < 3; i++) {
        Q<C> SB = {(C)0, (C)0, (C)0, (C)0};
#pragma unroll
        for (int j = 0; j < 3; j++) {
            if (j == i || (CARRY && j == 0)) continue;
            const Q<C> B = qmul(qmul(q(j, n.m[j]), qconj(q(i, n.m[j]))), qconj(q(j, n.dg(i, j))));
            SB = qadd_scaled(SB, l[j], B);
        }
        C b1, b2, b3;
        qmul_vec(U[i], SB, b1, b2, b3);
        Mg[i][0] -= b1;
        Mg[i][1] -= b2;
        Mg[i][2] -= b3;
    }
}

// What the site at n.c hands to its +x neighbour (XCarry), without evolving it:
// the start of an x-march, and sites on Fixed x faces.  Reads the planes x and x + 1.
template <class C, int ND, class A, class R>
__device__ __forceinline__ void site_carry(const A& acc, const Stencil<R>& n, XCarry<C, ND>& carry)
{
    const Q<C> U0 = acc.q(0, n.c);
    const C th0 = acc.th(0, n.c);
    C vj[3];
    plaq_forces(acc.q(1, n.p[0]), acc.q(0, n.p[1]), U0, acc.q(1, n.c), carry.v01, vj);
    plaq_forces(acc.q(2, n.p[0]), acc.q(0, n.p[2]), U0, acc.q(2, n.c), carry.v02, vj);
    carry.s01 = gsin(th0 + acc.th(1, n.p[0]) - acc.th(0, n.p[1]) - acc.th(1, n.c));
    carry.s02 = gsin(th0 + acc.th(2, n.p[0]) - acc.th(0, n.p[2]) - acc.th(2, n.c));
    C sn, cs;
    gsincos(th0, sn, cs);
#pragma unroll
    for (int db = 0; db < ND; db++) carry.t0[db] = transport(U0, cs, sn, acc.ph(db, n.c));
}

// asin of the three U(1) increments: the series where all are small, which
// the link update's increments are; one test for the three.
template <class C>
__device__ __forceinline__ void asin3(const C (&r)[3], C (&a)[3], unsigned& warn)
{
    MaxAbs<C> m;
#pragma unroll
    for (int d = 0; d < 3; d++) m.add(r[d]);
    if (m.exceeds(AsinSeries<C>::limit)) {
#pragma unroll
        for (int d = 0; d < 3; d++) {
            if (r[d] * r[d] > (C)1) warn |= kWarnAsin;
            a[d] = gasin(r[d]);
        }
    } else {
#pragma unroll
        for (int d = 0; d < 3; d++) a[d] = asin_series(r[d]);
    }
}

// Phases beyond the reduction range of the elementary functions.
template <class C>
__device__ __forceinline__ void warn_range(const C (&th)[3], unsigned& warn)
{
    MaxAbs<C> m;
#pragma unroll
    for (int d = 0; d < 3; d++) m.add(th[d]);
    if (m.exceeds((C)1e4)) {
#pragma unroll
        for (int d = 0; d < 3; d++)
            if (fabs(th[d]) > (C)1e4) warn |= kWarnRange;
    }
}

// dt^2 times a site's own-site scalar terms into D -- the Laplacian's diagonal minus dV/dphi, both
// multiples of the doublets -- and, on logging steps, its potential energy.
template <int MODEL, bool ENERGY, class C, int ND>
__device__ __forceinline__ double site_potential(const StepParams& P, const KConst<C>& F, const Q<C> (&fc)[ND],
                                                 Q<C> (&D)[ND])
{
    double pot_e = 0.0;
    if (MODEL == kModelSM) {
        const C fsq = fc[0].w * fc[0].w + fc[0].x * fc[0].x + fc[0].y * fc[0].y + fc[0].z * fc[0].z;
        const C k = F.diag + (F.rest - F.lambda * (fsq - F.eta_sqr));
        D[0] = {k * fc[0].w, k * fc[0].x, k * fc[0].y, k * fc[0].z};
        if (ENERGY) {
            const double t = (double)fsq - P.eta_sqr;
            pot_e = 0.25 * P.lambda * t * t;
        }
    } else {
        const Q<C> f1 = fc[0], f2 = fc[ND - 1];
        const C s1 = f1.w * f1.w + f1.x * f1.x + f1.y * f1.y + f1.z * f1.z;
        const C s2 = f2.w * f2.w + f2.x * f2.x + f2.y * f2.y + f2.z * f2.z;
        const C dot = P.break_son ? f1.w * f2.w + f1.x * f2.x + f1.y * f2.y + f1.z * f2.z : (C)0;
        const C anti = (P.break_son && P.break_uhalfn) ? f1.w * f2.x - f1.x * f2.w + f1.y * f2.z - f1.z * f2.y : (C)0;
        C a1 = F.m1x2 - F.l1x4 * s1 - F.l3x2 * s2;
        C a2 = F.m2x2 - F.l2x4 * s2 - F.l3x2 * s1;
        const C f1v[4] = {f1.w, f1.x, f1.y, f1.z};
        const C f2v[4] = {f2.w, f2.x, f2.y, f2.z};
        C v1[4], v2[4];
        if (P.break_son) {
            // single SO(N): (-m12r + 2 l4p5 dot + l6r s1 + l7r s2) f_other + 2 l6r|l7r dot f_self
            const C bs = F.m12r - F.l4p5x2 * dot - F.l6r * s1 - F.l7r * s2;
            a1 -= F.l6rx2 * dot;
            a2 -= F.l7rx2 * dot;
            if (P.break_uhalfn) {
                // U(N/2): (m12i + 2 l4m5 anti - 2 l5i dot - l6i s1 - l7i s2) J f_other - 2 l5i anti f_other
                // - 2 l6i|l7i anti f_self
                const C cu = F.l5ix2 * dot + F.l6i * s1 + F.l7i * s2 - F.m12i - F.l4m5x2 * anti;
                const C bo = bs + F.l5ix2 * anti;
                a1 = F.diag + (a1 + F.l6ix2 * anti);
                a2 = F.diag + (a2 + F.l7ix2 * anti);
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    const int alt = 1 - 2 * (k % 2);
                    v1[k] = a1 * f1v[k] + bo * f2v[k] + cu * (C)alt * f2v[k + alt];
                    v2[k] = a2 * f2v[k] + bo * f1v[k] - cu * (C)alt * f1v[k + alt];
                }
            } else {
                a1 += F.diag;
                a2 += F.diag;
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    v1[k] = a1 * f1v[k] + bs * f2v[k];
                    v2[k] = a2 * f2v[k] + bs * f1v[k];
                }
            }
        } else {
            a1 += F.diag;
            a2 += F.diag;
#pragma unroll
            for (int k = 0; k < 4; k++) {
                v1[k] = a1 * f1v[k];
                v2[k] = a2 * f2v[k];
            }
        }
        D[0] = {v1[0], v1[1], v1[2], v1[3]};
        D[ND - 1] = {v2[0], v2[1], v2[2], v2[3]};
        if (ENERGY) {
            const double d1 = s1, d2 = s2, dd = dot, da = anti;
            double v = -P.m1 * d1 - P.m2 * d2 + P.l1 * d1 * d1 + P.l2 * d2 * d2 + P.l3 * d1 * d2;
            if (P.break_son) {
                v += -P.m12r * dd + P.l4p5 * dd * dd + P.l6r * d1 * dd + P.l7r * d2 * dd;
                if (P.break_uhalfn)
                    v += P.m12i * da + P.l4m5 * da * da - 2.0 * P.l5i * dd * da - P.l6i * d1 * da - P.l7i * d2 * da;
            }
            if (P.apply_norm) v += P.energy_offset;
            pot_e = v;
        }
    }
    return pot_e;
}

// Scalar leapfrog (Model.cpp:347-356) of one doublet f, from D = dt^2 (Laplacian - dV/dphi):
// phi(t+dt) = phi + [(phi - phi_past)(1 - damping) + D], one rounding at the end.
template <bool ENERGY, class C, class S>
__device__ __forceinline__ void leapfrog_doublet(const KConst<C>& F, Q<C> f, Q<C> fpast, Q<C> D, S* out, int s, C& kin_e,
                                                 C& phisq, C& check)
{
    const C fn[4] = {f.w, f.x, f.y, f.z};
    const C fo[4] = {fpast.w, fpast.x, fpast.y, fpast.z};
    const C dd[4] = {D.w, D.x, D.y, D.z};
    C o[4];
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const C vel = fn[k] - fo[k];
        o[k] = fn[k] + (F.keep * vel + dd[k]);
        check += o[k];
        if (ENERGY) {
            kin_e += vel * vel;  // x 0.5 / dt^2 in record_energies
            phisq += fn[k] * fn[k];
        }
    }
    st4(out, s, o[0], o[1], o[2], o[3]);
}

// Link update (WilsonLoops/Source/StandardModel.cpp:456-514) from the forces dt^2 (magnetic + current).
template <bool ENERGY, class C, class PV>
__device__ __forceinline__ void leapfrog_links(const KConst<C>& F, const Q<C> (&U)[3], const C (&th)[3],
                                               const C (&Mg)[3][3], const C (&MgY)[3], const PV& past, C& elec_e,
                                               unsigned& warn, C& check)
{
    // theta(t+dt) = theta(t) + asin(RHS_Y)
    C R0[3], inc[3];
#pragma unroll
    for (int d = 0; d < 3; d++) {
        const C dth = th[d] - past.th(d);
        R0[d] = F.keep * gsin(dth) + MgY[d];
        if (ENERGY) {  // 1 - cos(dtheta) = 2 sin^2(dtheta/2)
            const C h = gsin((C)0.5 * dth);
            elec_e += F.e_elec[d] * (F.inv_gp_sqr * (C)2 * h * h);
        }
    }
    warn_range(th, warn);
    asin3(R0, inc, warn);
#pragma unroll
    for (int d = 0; d < 3; d++) {
        const C thn = th[d] + inc[d];
        check += thn;
        past.at.L.th[d][past.at.s] = thn;
    }
    // u = (sqrt(1-|c|^2), c); U(t+dt) = normalise(u U(t)) (su2_advance3)
    C W[3][3];
#pragma unroll
    for (int d = 0; d < 3; d++) {
        const Q<C> Un = U[d];
        const Q<C> Up = past.q(d);
        // link momentum vec(U_now U_past^dag) = vec((U_now - U_past) U_past^dag)
        const Q<C> dlt = {Un.w - Up.w, Un.x - Up.x, Un.y - Up.y, Un.z - Up.z};
        C E1, E2, E3;
        qmul_vec(dlt, qconj(Up), E1, E2, E3);
        W[d][0] = F.keep * E1 + Mg[d][0];
        W[d][1] = F.keep * E2 + Mg[d][1];
        W[d][2] = F.keep * E3 + Mg[d][2];
        if (ENERGY) {
            // 1 - (U_now U_past^dag)_0 / |U_now U_past^dag|
            const Q<C> Ed = {Un.w * Up.w + Un.x * Up.x + Un.y * Up.y + Un.z * Up.z, E1, E2, E3};
            elec_e += F.e_elec[d] * (F.inv_g_sqr * one_minus_trace(Ed));
        }
    }
    su2_advance3(U, W, past.at.L.q, past.at.s, warn, check);
}

// A site's energy densities into the thread's sums, and into the local output where it is asked for.
template <class C>
__device__ __forceinline__ void record_energies(const StepParams& P, int s, double pot_e, C grad_e, C kin_e, C mag_e,
                                                C elec_e, C plaq2, C plaq1, C phisq, double (&obs)[kObsCount])
{
    const double ge = (double)grad_e, ke = 0.5 * P.inv_sqr_dt * (double)kin_e;
    const double me = (double)mag_e, ee = (double)elec_e;
    if (P.loc_energy) {  // Energy's local densities (Analysers/Source/Energy.cpp:137-143)
        float* o = P.loc_energy + 6 * (size_t)s;
        o[0] = (float)(pot_e + ge + ke + me + ee);
        o[1] = (float)pot_e;
        o[2] = (float)ge;
        o[3] = (float)ke;
        o[4] = (float)me;
        o[5] = (float)ee;
    }
    obs[kObsPotential] += pot_e;
    obs[kObsGradient] += ge;
    obs[kObsKinetic] += ke;
    obs[kObsMagnetic] += me;
    obs[kObsElectric] += ee;
    obs[kObsPlaqSU2] += (double)plaq2;
    obs[kObsPlaqU1] += (double)plaq1;
    obs[kObsPhiSq] += (double)phisq;
}

// The per-site update.  A provides q(d, R) -> Q<C>, th(d, R) -> C, ph(k, R) -> Q<C>
// for the "now" level (and hth / hq for a 2HDM Higgs-family field, HF != 0).
// obs receives the energy-step observables except the total (energy_total after
// the last site) and warn the warning bits, both only when `count` (the site is
// not on a ghost plane).  CARRY (HF == 0 only): `carry` holds the x - 1 site's
// values (site_step or site_carry of that site) and receives this site's; nothing
// of the plane x - 1 is read.  Forces are formed already multiplied by dt^2 (the
// constants of KConst).
template <class S, int MODEL, bool ENERGY, int HF = kHfNone, bool CARRY = false, class A, class R, class LV>
__device__ __forceinline__ void site_step(const StepParams& P, const KConst<S>& F, const A& acc, const Stencil<R>& n,
                                          PastSite<S, LV> ps,
                                          XCarry<S, (MODEL == kModelSM) ? 1 : 2>& carry, double (&obs)[kObsCount],
                                          unsigned& warn, bool count = true)
{
    static_assert(!CARRY || HF == kHfNone, "the x-carry holds no Higgs-family values");
    const unsigned warn_in = warn;
    using C = S;  // FP64 form -> double, mixed form -> float
    constexpr int ND = (MODEL == kModelSM) ? 1 : 2;
    PastValues<S, ND, LV, !ENERGY> past = {ps};
    past.load();
    const C l[3] = {F.ldt[0], F.ldt[1], F.ldt[2]};  // dt^2 / dx_a^2

    Q<C> U[3];
    C th[3];
#pragma unroll
    for (int a = 0; a < 3; a++) {
        U[a] = acc.q(a, n.c);
        th[a] = acc.th(a, n.c);
    }

    // ---- magnetic term: U(1) sines and SU(2) loops ----
    // logging-step terms: per-site partial sums in the form's arithmetic (a few
    // cancellation-free terms each), added to the FP64 block sums once per site
    C mag_e = (C)0, plaq2 = (C)0, plaq1 = (C)0;
    // F_ij(x) = theta_i(x) + theta_j(x+i) - theta_i(x+j) - theta_j(x) of the upper loops; the
    // reference's local angle is -F for link i and +F for link j (StandardModel.cpp:348-353).
    // Then the lower loops' angles, those of the planes with x carried as sines.
    constexpr int NLOW = CARRY ? 4 : 6;
    C Fa[3 + NLOW], sF[3 + NLOW];
#pragma unroll
    for (int pl = 0; pl < 3; pl++) {
        const int i = (pl == 2) ? 1 : 0;
        const int j = (pl == 0) ? 1 : 2;
        Fa[pl] = th[i] + acc.th(j, n.p[i]) - acc.th(i, n.p[j]) - th[j];
    }
    {
        int k = 3;
#pragma unroll
        for (int i = 0; i < 3; i++) {
#pragma unroll
            for (int j = 0; j < 3; j++) {
                if (j == i || (CARRY && j == 0)) continue;
                const R mj = n.m[j];
                Fa[k++] = -acc.th(j, n.dg(i, j)) - acc.th(i, mj) + acc.th(j, mj) + th[i];
            }
        }
    }
#pragma unroll
    for (int k = 0; k < 3 + NLOW; k++) sF[k] = gsin(Fa[k]);
    C MgY[3];
    MgY[0] = -l[1] * sF[0] - l[2] * sF[1];
    MgY[1] = l[0] * sF[0] - l[2] * sF[2];
    MgY[2] = l[0] * sF[1] + l[1] * sF[2];
    if constexpr (CARRY) {
        MgY[1] -= l[0] * carry.s01;
        MgY[2] -= l[0] * carry.s02;
        carry.s01 = sF[0];
        carry.s02 = sF[1];
    }
    {
        int k = 3;
#pragma unroll
        for (int i = 0; i < 3; i++) {
#pragma unroll
            for (int j = 0; j < 3; j++) {
                if (j == i || (CARRY && j == 0)) continue;
                MgY[i] -= sF[k++] * l[j];
            }
        }
    }
    if (ENERGY) {
#pragma unroll
        for (int pl = 0; pl < 3; pl++) {
            // 1 - cos F = 2 sin^2(F/2) (no cancellation for small F)
            const C hF = gsin((C)0.5 * Fa[pl]);
            const C omc = (C)2 * hF * hF;
            mag_e += F.e_plaq[pl] * (F.inv_gp_sqr * omc);
            plaq1 += (C)1 - omc;
        }
    }
    C Mg[3][3];
    su2_force<CARRY>([&](int d, const R& r) { return acc.q(d, r); }, n, U, l, carry.v01, carry.v02, Mg,
                     [&](int pl, Q<C> p) {
                         if (ENERGY) {
                             const C omt = one_minus_trace(p);
                             mag_e += F.e_plaq[pl] * (F.inv_g_sqr * omt);
                             plaq2 += (C)1 - omt;
                         }
                     });
    // ---- Higgs-family magnetic term (WilsonLoops/Source/TwoHDM.cpp:484-551): the same
    //      loops on theta_H (U(1)) or the family quaternion (SU(2)), coupling g'' ----
    C MgH[3][3];
#pragma unroll
    for (int i = 0; i < 3; i++) MgH[i][0] = MgH[i][1] = MgH[i][2] = (C)0;
    if constexpr (HF == kHfU1) {
        C hc[3];
#pragma unroll
        for (int a = 0; a < 3; a++) hc[a] = acc.hth(a, n.c);
#pragma unroll
        for (int pl = 0; pl < 3; pl++) {
            const int i = (pl == 2) ? 1 : 0;
            const int j = (pl == 0) ? 1 : 2;
            const C Fa = hc[i] + acc.hth(j, n.p[i]) - acc.hth(i, n.p[j]) - hc[j];
            const C sF = gsin(Fa);
            MgH[i][0] -= sF * l[j];
            MgH[j][0] += sF * l[i];
            if (ENERGY) {
                const C hF = gsin((C)0.5 * Fa);
                mag_e += F.e_plaq[pl] * F.inv_gpp_sqr * ((C)2 * hF * hF);
            }
        }
#pragma unroll
        for (int i = 0; i < 3; i++) {
#pragma unroll
            for (int j = 0; j < 3; j++) {
                if (j == i) continue;
                const C neigh = -acc.hth(j, n.dg(i, j)) - acc.hth(i, n.m[j]) + acc.hth(j, n.m[j]) + hc[i];
                MgH[i][0] -= gsin(neigh) * l[j];
            }
        }
    } else if constexpr (HF == kHfSU2) {
        Q<C> UH[3];
#pragma unroll
        for (int a = 0; a < 3; a++) UH[a] = acc.hq(a, n.c);
        su2_force<false>([&](int d, const R& r) { return acc.hq(d, r); }, n, UH, l, carry.v01, carry.v02, MgH,
                         [&](int pl, Q<C> p) {
                             if (ENERGY) mag_e += F.e_plaq[pl] * F.inv_gpp_sqr * one_minus_trace(p);
                         });
    }

    // ---- potential dV/dphi and the Laplacian's diagonal ----
    Q<C> fc[ND];
#pragma unroll
    for (int db = 0; db < ND; db++) fc[db] = acc.ph(db, n.c);
    Q<C> D[ND];
    const double pot_e = site_potential<MODEL, ENERGY>(P, F, fc, D);

    // ---- scalar sector: covariant Laplacian D and currents J (four times the reference's, whose
    //      1/4 is in the constants cY, cI and cH; the SU(2) currents join Mg) ----
    C JY[3];
    C JH[3][3];  // Higgs-family currents (Gradients/Source/TwoHDM.cpp:465-485)
    C grad_e = (C)0;
    constexpr int A0 = CARRY ? 1 : 0;  // directions whose backward transport is computed (x's is carried)
    C ang[6 - A0], sn[6 - A0], cs[6 - A0];
#pragma unroll
    for (int a = 0; a < 3; a++) {
        ang[a] = th[a];
        if (a >= A0) ang[3 + a - A0] = acc.th(a, n.m[a]);
    }
#pragma unroll
    for (int k = 0; k < 6 - A0; k++) gsincos(ang[k], sn[k], cs[k]);
#pragma unroll
    for (int a = 0; a < 3; a++) {
        const bool back = a >= A0;
        // The doublet transported forward, U R phi: what the next site of a march and the family
        // currents need.  Elsewhere the current is formed from phi and the transported-back
        // neighbour and turned by the link.
        const bool fwd = HF != kHfNone || !back;
        Q<C> tm[ND], tp[ND], t[ND], fp[ND];
#pragma unroll
        for (int db = 0; db < ND; db++) {
            fp[db] = acc.ph(db, n.p[a]);
            // D: U_a(x-a) phi(x-a) + U_a(x)^dag phi(x+a); the first is the x-1 site's transported doublet
            tm[db] = back ? transport(acc.q(a, n.m[a]), cs[3 + a - A0], sn[3 + a - A0], acc.ph(db, n.m[a]))
                          : carry.t0[db];
            tp[db] = transport_back(U[a], cs[a], sn[a], fp[db]);
            t[db] = fwd ? transport(U[a], cs[a], sn[a], fc[db]) : fc[db];
            if (!back) carry.t0[db] = t[db];
        }
        if constexpr (HF == kHfU1) {
            C hsn, hcs, hsm, hcm;
            gsincos(acc.hth(a, n.c), hsn, hcs);
            gsincos(acc.hth(a, n.m[a]), hsm, hcm);
            const Q<C> one = {(C)1, (C)0, (C)0, (C)0};
            hf_act<HF>(tm[0], tm[1], hcm, hsm, one);
            hf_act<HF>(tp[0], tp[1], hcs, -hsn, one);
            hf_act<HF>(t[0], t[1], hcs, hsn, one);
        } else if constexpr (HF == kHfSU2) {
            const Q<C> uh = acc.hq(a, n.c), uhm = acc.hq(a, n.m[a]);
            hf_act<HF>(tm[0], tm[1], (C)1, (C)0, uhm);
            hf_act<HF>(tp[0], tp[1], (C)1, (C)0, qconj(uh));
            hf_act<HF>(t[0], t[1], (C)1, (C)0, uh);
        }
        C J[3];
#pragma unroll
        for (int db = 0; db < ND; db++) {
            D[db] = qadd_scaled(D[db], l[a], tm[db]);
            D[db] = qadd_scaled(D[db], l[a], tp[db]);
            // J: Im of t^dag sigma f, with t = U phi and f = phi(x+a), or phi and U^dag phi(x+a)
            const Q<C> u = t[db], f = fwd ? fp[db] : tp[db];
            const C up = u.w * f.x - u.x * f.w, lo = u.y * f.z - u.z * f.y;
            const C j1 = u.w * f.z - u.x * f.y + u.y * f.x - u.z * f.w;
            const C j2 = -u.w * f.y - u.x * f.z + u.y * f.w + u.z * f.x;
            JY[a] = (db ? JY[a] : (C)0) + (up + lo);
            J[0] = (db ? J[0] : (C)0) + j1;
            J[1] = (db ? J[1] : (C)0) + j2;
            J[2] = (db ? J[2] : (C)0) + (up - lo);
            if (ENERGY) {
                const C e0 = f.w - u.w, e1 = f.x - u.x, e2 = f.y - u.y, e3 = f.z - u.z;
                grad_e += F.e_grad[a] * (e0 * e0 + e1 * e1 + e2 * e2 + e3 * e3);
            }
        }
        if (fwd) {
#pragma unroll
            for (int k = 0; k < 3; k++) Mg[a][k] += F.cI * J[k];
        } else {
            add_turned(Mg[a], F.cI, U[a], J);
        }
        if constexpr (HF != kHfNone) {
            // family pairs: components (i, i+1) of doublet 1 and of doublet 2, i = 0 (upper) and 2 (lower)
            const C t8[8] = {t[0].w, t[0].x, t[0].y, t[0].z, t[1].w, t[1].x, t[1].y, t[1].z};
            const C n8[8] = {fp[0].w, fp[0].x, fp[0].y, fp[0].z, fp[1].w, fp[1].x, fp[1].y, fp[1].z};
            C h4 = 0, h5 = 0, h6 = 0;
#pragma unroll
            for (int i = 0; i < 4; i += 2) {
                if constexpr (HF == kHfU1) {
                    h4 += t8[i] * n8[i + 1] - t8[i + 1] * n8[i] - t8[i + 4] * n8[i + 5] + t8[i + 5] * n8[i + 4];
                } else {
                    h4 += t8[i] * n8[i + 5] - t8[i + 1] * n8[i + 4] + t8[i + 4] * n8[i + 1] - t8[i + 5] * n8[i];
                    h5 += -t8[i] * n8[i + 4] - t8[i + 1] * n8[i + 5] + t8[i + 4] * n8[i] + t8[i + 5] * n8[i + 1];
                    h6 += t8[i] * n8[i + 1] - t8[i + 1] * n8[i] - t8[i + 4] * n8[i + 5] + t8[i + 5] * n8[i + 4];
                }
            }
            JH[a][0] = h4;
            JH[a][1] = h5;
            JH[a][2] = h6;
        }
    }

    C kin_e = (C)0, phisq = (C)0, elec_e = (C)0;
    C check = (C)0;  // sum of every new value: non-finite iff one of them is
    const C keep = F.keep;
#pragma unroll
    for (int db = 0; db < ND; db++)
        leapfrog_doublet<ENERGY>(F, fc[db], past.ph(db), D[db], ps.L.ph[db], ps.s, kin_e, phisq, check);
#pragma unroll
    for (int d = 0; d < 3; d++) MgY[d] += F.cY * JY[d];
    leapfrog_links<ENERGY>(F, U, th, Mg, MgY, past, elec_e, warn, check);

    // Higgs-family links (WilsonLoops/Source/TwoHDM.cpp:601-633, 702-745), coupling g''
    if constexpr (HF == kHfU1) {
        C RH[3], hinc[3], hn[3];
#pragma unroll
        for (int d = 0; d < 3; d++) {
            hn[d] = acc.hth(d, n.c);
            const C dh = hn[d] - ld1<C>(ps.L.hth[d], ps.s);
            RH[d] = keep * gsin(dh) + (MgH[d][0] + F.cH * JH[d][0]);
            if (ENERGY) {
                const C h = gsin((C)0.5 * dh);
                elec_e += F.e_elec[d] * F.inv_gpp_sqr * ((C)2 * h * h);
            }
        }
        warn_range(hn, warn);
        asin3(RH, hinc, warn);
#pragma unroll
        for (int d = 0; d < 3; d++) {
            const C hnew = hn[d] + hinc[d];
            check += hnew;
            ps.L.hth[d][ps.s] = hnew;
        }
    } else if constexpr (HF == kHfSU2) {
        Q<C> H[3];
        C RH[3][3];
#pragma unroll
        for (int d = 0; d < 3; d++) {
            const Q<C> Hn = acc.hq(d, n.c);
            H[d] = Hn;
            const Q<C> Hp = ld4<C>(ps.L.hq[d], ps.s);
            const Q<C> dH = {Hn.w - Hp.w, Hn.x - Hp.x, Hn.y - Hp.y, Hn.z - Hp.z};
            C F1, F2, F3;
            qmul_vec(dH, qconj(Hp), F1, F2, F3);
            RH[d][0] = keep * F1 + (MgH[d][0] + F.cH * JH[d][0]);
            RH[d][1] = keep * F2 + (MgH[d][1] + F.cH * JH[d][1]);
            RH[d][2] = keep * F3 + (MgH[d][2] + F.cH * JH[d][2]);
            if (ENERGY) {
                const Q<C> Ed = {Hn.w * Hp.w + Hn.x * Hp.x + Hn.y * Hp.y + Hn.z * Hp.z, F1, F2, F3};
                elec_e += F.e_elec[d] * F.inv_gpp_sqr * one_minus_trace(Ed);
            }
        }
        su2_advance3(H, RH, ps.L.hq, ps.s, warn, check);
    }
    if (!isfinite(check)) warn |= kWarnNonFinite;
    if (!count) {
        warn = warn_in;
        return;
    }

    if (ENERGY) record_energies(P, ps.s, pot_e, grad_e, kin_e, mag_e, elec_e, plaq2, plaq1, phisq, obs);
}

// Gauss-law residual at site c after a step (Analysers/Source/GaugeCondition.cpp:117-165,
// Core/Source/Model.cpp:323-337 semantics), in FP64 for every form; md[a] is
// the site x - e_a.  v[k] = v[4 + k] = |violation of constraint k| (the
// integrated and the maximum slot of the analyser).  sin is the library's
// double series.
// One link direction at one site, both levels, as FP64 values.
struct GLink {
    Q<double> now, fut;
    double tnow, tfut;
};

template <class S, class LV>
__device__ __forceinline__ GLink gauss_link(const LV& now, const LV& fut, int d, int s)
{
    return {ld4<double>(now.q[d], s), ld4<double>(fut.q[d], s), ld1<double>(now.th[d], s), ld1<double>(fut.th[d], s)};
}

// The residuals from the links at x (own[d]) and at x - e_d (back[d]) and the
// doublets at x (phn / phf: both levels; site c for the local output).
// NEQ_ALL: the local-violation stride (gaugeNum; the Higgs-family constraints follow)
template <int MODEL, int NEQ_ALL = 4>
__device__ __forceinline__ void gauss_core(const StepParams& P, const GLink (&own)[3], const GLink (&back)[3],
                                           const Q<double> (&phn)[2], const Q<double> (&phf)[2], int c,
                                           double (&v)[kGaussSlots])
{
    constexpr int ND = (MODEL == kModelSM) ? 1 : 2;
    double el[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
    for (int d = 0; d < 3; d++) {
        const double la = own[d].tfut - own[d].tnow;
        const double na = back[d].tfut - back[d].tnow;
        el[0] += (gsin(la) - gsin(na)) * P.lap[d];
        // vec(U_now(x)^dag U_fut(x)) - vec(U_fut(x-d) U_now(x-d)^dag)
        double a1, a2, a3, b1, b2, b3;
        qmul_vec(qconj(own[d].now), own[d].fut, a1, a2, a3);
        qmul_vec(back[d].fut, qconj(back[d].now), b1, b2, b3);
        el[1] += (a1 - b1) * P.lap[d];
        el[2] += (a2 - b2) * P.lap[d];
        el[3] += (a3 - b3) * P.lap[d];
    }
    double gr[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
    for (int db = 0; db < ND; db++) {
        const Q<double> p = phn[db];
        const Q<double> q = phf[db];
        gr[0] += 0.25 * (p.w * q.x - p.x * q.w + p.y * q.z - p.z * q.y);
        gr[1] += 0.25 * (p.w * q.z - p.x * q.y + p.y * q.x - p.z * q.w);
        gr[2] += 0.25 * (-p.w * q.y - p.x * q.z + p.y * q.w + p.z * q.x);
        gr[3] += 0.25 * (p.w * q.x - p.x * q.w - p.y * q.z + p.z * q.y);
    }
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const double viol = el[k] - P.gsq[k] * gr[k];
        const double av = fabs(viol);
        v[k] = av;
        v[4 + k] = av;
        if (P.loc_gauss) P.loc_gauss[(size_t)NEQ_ALL * c + k] = (float)viol;  // GaugeCondition local violation
    }
}

// v = |violation| of the 2 * gaugeNum slots (integrated then maximum) per
// constraint; with a Higgs-family field (HF != 0) the constraints 4.. of
// WilsonLoops/Source/TwoHDM.cpp:357-392 and Gradients/Source/TwoHDM.cpp:355-372 follow.
template <class S, int MODEL, int HF = kHfNone, class LV>
__device__ __forceinline__ void gauss_site(const StepParams& P, const LV& now, const LV& fut,
                                           int c, int md0, int md1, int md2, double (&v)[2 * hf_neq(HF)])
{
    const GLink own[3] = {gauss_link<S>(now, fut, 0, c), gauss_link<S>(now, fut, 1, c), gauss_link<S>(now, fut, 2, c)};
    const GLink back[3] = {gauss_link<S>(now, fut, 0, md0), gauss_link<S>(now, fut, 1, md1), gauss_link<S>(now, fut, 2, md2)};
    Q<double> phn[2], phf[2];
#pragma unroll
    for (int db = 0; db < ((MODEL == kModelSM) ? 1 : 2); db++) {
        phn[db] = ld4<double>(now.ph[db], c);
        phf[db] = ld4<double>(fut.ph[db], c);
    }
    if constexpr (HF == kHfNone) {
        gauss_core<MODEL>(P, own, back, phn, phf, c, v);
    } else {
        constexpr int NEQ = hf_neq(HF);
        double vs[kGaussSlots];
        gauss_core<MODEL, NEQ>(P, own, back, phn, phf, c, vs);
#pragma unroll
        for (int k = 0; k < 4; k++) {
            v[k] = vs[k];
            v[NEQ + k] = vs[4 + k];
        }
        const int md[3] = {md0, md1, md2};
        double el[3] = {0.0, 0.0, 0.0};
#pragma unroll
        for (int d = 0; d < 3; d++) {
            if constexpr (HF == kHfU1) {
                const double la = ld1<double>(fut.hth[d], c) - ld1<double>(now.hth[d], c);
                const double na = ld1<double>(fut.hth[d], md[d]) - ld1<double>(now.hth[d], md[d]);
                el[0] += (gsin(la) - gsin(na)) * P.lap[d];
            } else {
                double a1, a2, a3, b1, b2, b3;
                qmul_vec(qconj(ld4<double>(now.hq[d], c)), ld4<double>(fut.hq[d], c), a1, a2, a3);
                qmul_vec(ld4<double>(fut.hq[d], md[d]), qconj(ld4<double>(now.hq[d], md[d])), b1, b2, b3);
                el[0] += (a1 - b1) * P.lap[d];
                el[1] += (a2 - b2) * P.lap[d];
                el[2] += (a3 - b3) * P.lap[d];
            }
        }
        const Q<double> p1 = ld4<double>(now.ph[0], c), p2 = ld4<double>(now.ph[1], c);
        const Q<double> q1 = ld4<double>(fut.ph[0], c), q2 = ld4<double>(fut.ph[1], c);
        const double a8[8] = {p1.w, p1.x, p1.y, p1.z, p2.w, p2.x, p2.y, p2.z};
        const double b8[8] = {q1.w, q1.x, q1.y, q1.z, q2.w, q2.x, q2.y, q2.z};
        double gr[3] = {0.0, 0.0, 0.0};
#pragma unroll
        for (int i = 0; i < 4; i += 2) {
            if constexpr (HF == kHfU1) {
                gr[0] += 0.25 * (a8[i] * b8[i + 1] - a8[i + 1] * b8[i] - a8[i + 4] * b8[i + 5] + a8[i + 5] * b8[i + 4]);
            } else {
                gr[0] += 0.25 * (a8[i] * b8[i + 5] - a8[i + 1] * b8[i + 4] + a8[i + 4] * b8[i + 1] - a8[i + 5] * b8[i]);
                gr[1] += 0.25 * (-a8[i] * b8[i + 4] - a8[i + 1] * b8[i + 5] + a8[i + 4] * b8[i] + a8[i + 5] * b8[i + 1]);
                gr[2] += 0.25 * (a8[i] * b8[i + 1] - a8[i + 1] * b8[i] - a8[i + 4] * b8[i + 5] + a8[i + 5] * b8[i + 4]);
            }
        }
#pragma unroll
        for (int k = 0; k < NEQ - 4; k++) {
            const double viol = el[k] - P.gsq_hf * gr[k];
            const double av = fabs(viol);
            v[4 + k] = av;
            v[NEQ + 4 + k] = av;
            if (P.loc_gauss) P.loc_gauss[(size_t)NEQ * c + 4 + k] = (float)viol;
        }
    }
}

}  // namespace gft
