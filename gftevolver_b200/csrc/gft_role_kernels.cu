// gft_role_kernels.cu -- the throughput forms' step for small lattices: a site's update
// divided over the warps of a block.
//
// A small lattice leaves most schedulers without a warp, and its step takes as long as
// one thread's chain of some 1,300 to 3,000 instructions.  Here a block takes 32 sites
// and one warp per part of their update, none of which waits for another:
//   roles 0-2: the SU(2) and U(1) link of direction d -- its loops, its current, its
//              momentum and update (and the 2HDM's family U(1) link);
//   role 3   : the doublets -- potential, covariant Laplacian, leapfrog;
//   roles 4-6: the family SU(2) link of direction d (gaugeNum 7).
// What two roles need (a transported doublet, a sine) both compute: a quarter more work
// in all, on schedulers that would idle.  The arithmetic is gft_step_body.cuh's.
#include "gft_device.cuh"
#include "gft_launch.h"
#include "gft_math.cuh"
#include "gft_step_body.cuh"

namespace gft {
namespace {

constexpr int role_count(int hf) { return hf == kHfSU2 ? 7 : 4; }

// Energies of a site, summed over its roles (the slots of a row but the total).
enum RoleSlot { kRPot, kRGrad, kRKin, kRMag, kRElec, kRPlaq2, kRPlaq1, kRPhiSq, kRCount };

// The site c and a link direction d with the other two, a < b: offsets to x +- e.
struct LinkSite {
    int c, d, a, b;
    int pd, pa, pb, ma, mb;
    __device__ __forceinline__ static void axis(const StepParams& P, int ax, int x, int y, int z, int& m, int& p)
    {
        const int n = (ax == 0) ? P.nx : (ax == 1 ? P.ny : P.nz);
        const int st = (ax == 0) ? P.ny * P.nz : (ax == 1 ? P.nz : 1);
        const int v = (ax == 0) ? x : (ax == 1 ? y : z);
        m = (v == 0) ? (n - 1) * st : -st;
        p = (v + 1 == n) ? -(n - 1) * st : st;
    }
    __device__ __forceinline__ LinkSite(const StepParams& P, int c, int d, int x, int y, int z) : c(c), d(d)
    {
        a = (d == 0) ? 1 : 0;
        b = (d == 2) ? 1 : 2;
        int md;
        axis(P, d, x, y, z, md, pd);
        axis(P, a, x, y, z, ma, pa);
        axis(P, b, x, y, z, mb, pb);
    }
};

// The SU(2) force on link d, dt^2-weighted, from the arrays q; with ENERGY the 1 - trace of its
// upper plaquettes, summed with their weights where the plane is counted here (the other
// direction is the higher one).
template <bool ENERGY, class S>
__device__ __forceinline__ void link_force(const KConst<S>& F, S* const* q, const LinkSite& n, Q<S> U, S (&M)[3],
                                           S& mag_e, S& plaq2, S weight)
{
    using C = S;
    Q<C> SB = {(C)0, (C)0, (C)0, (C)0};
#pragma unroll
    for (int k = 0; k < 3; k++) M[k] = (C)0;
#pragma unroll
    for (int o = 0; o < 2; o++) {
        const int j = o ? n.b : n.a, pj = o ? n.pb : n.pa, mj = o ? n.mb : n.ma;
        const C l = F.ldt[j];
        C vi[3], vj[3];
        const C w = plaq_forces(ld4<C>(q[j], n.c + n.pd), ld4<C>(q[n.d], n.c + pj), U, ld4<C>(q[j], n.c), vi, vj);
#pragma unroll
        for (int k = 0; k < 3; k++) M[k] += l * vi[k];
        if (ENERGY && n.d < j) {
            const C omt = one_minus_trace(Q<C>{w, vi[0], vi[1], vi[2]});
            mag_e += F.e_plaq[n.d + j - 1] * weight * omt;
            plaq2 += (C)1 - omt;
        }
        const Q<C> B = qmul(qmul(ld4<C>(q[j], n.c + mj), qconj(ld4<C>(q[n.d], n.c + mj))),
                            qconj(ld4<C>(q[j], n.c + n.pd + mj)));
        SB = qadd_scaled(SB, l, B);
    }
    C b1, b2, b3;
    qmul_vec(U, SB, b1, b2, b3);
    M[0] -= b1;
    M[1] -= b2;
    M[2] -= b3;
}

// The same for a U(1) link from the phases th.
template <bool ENERGY, class S>
__device__ __forceinline__ S phase_force(const KConst<S>& F, S* const* th, const LinkSite& n, S td, S& mag_e, S& plaq1,
                                         S weight)
{
    using C = S;
    C m = (C)0;
#pragma unroll
    for (int o = 0; o < 2; o++) {
        const int j = o ? n.b : n.a, pj = o ? n.pb : n.pa, mj = o ? n.mb : n.ma;
        const C up = td + ld1<C>(th[j], n.c + n.pd) - ld1<C>(th[n.d], n.c + pj) - ld1<C>(th[j], n.c);
        const C lo = -ld1<C>(th[j], n.c + n.pd + mj) - ld1<C>(th[n.d], n.c + mj) + ld1<C>(th[j], n.c + mj) + td;
        m -= F.ldt[j] * (gsin(up) + gsin(lo));
        if (ENERGY && n.d < j) {
            const C h = gsin((C)0.5 * up), omc = (C)2 * h * h;
            mag_e += F.e_plaq[n.d + j - 1] * weight * omc;
            plaq1 += (C)1 - omc;
        }
    }
    return m;
}

// New SU(2) link from its dt^2-weighted force M (su2_advance3's formula for one link).
template <bool ENERGY, class S>
__device__ __forceinline__ void advance_link(const KConst<S>& F, S* out, int s, Q<S> Un, Q<S> Up, const S (&M)[3],
                                             S weight, S& elec_e, unsigned& warn, S& check)
{
    using C = S;
    const Q<C> dlt = {Un.w - Up.w, Un.x - Up.x, Un.y - Up.y, Un.z - Up.z};
    C E1, E2, E3;
    qmul_vec(dlt, qconj(Up), E1, E2, E3);
    const C R1 = F.keep * E1 + M[0], R2 = F.keep * E2 + M[1], R3 = F.keep * E3 + M[2];
    if (ENERGY) {
        const Q<C> Ed = {Un.w * Up.w + Un.x * Up.x + Un.y * Up.y + Un.z * Up.z, E1, E2, E3};
        elec_e += weight * one_minus_trace(Ed);
    }
    const C cm = R1 * R1 + R2 * R2 + R3 * R3;
    if (cm > (C)1) warn |= kWarnSqrt;
    C e = fma(Un.w, Un.w, (C)-1);
    e = fma(Un.x, Un.x, e);
    e = fma(Un.y, Un.y, e);
    e = fma(Un.z, Un.z, e);
    const C f = e * ((C)0.375 * e - (C)0.5), u0m1 = sqrt1m_minus1(cm), a = fma(f, u0m1, u0m1 + f);
    const Q<C> dU = qmul(Q<C>{a, fma(f, R1, R1), fma(f, R2, R2), fma(f, R3, R3)}, Un);
    check += a;
    st4(out, s, Un.w + dU.w, Un.x + dU.x, Un.y + dU.y, Un.z + dU.z);
}

template <bool ENERGY, class S>
__device__ __forceinline__ void advance_phase(const KConst<S>& F, S* out, int s, S tn, S tp, S M, S weight, S& elec_e,
                                              unsigned& warn, S& check)
{
    const S dth = tn - tp;
    const S R = F.keep * gsin(dth) + M;
    if (ENERGY) {
        const S h = gsin((S)0.5 * dth);
        elec_e += weight * ((S)2 * h * h);
    }
    if (R * R > (S)1) warn |= kWarnAsin;
    if (fabs(tn) > (S)1e4) warn |= kWarnRange;
    const S v = tn + gasin(R);
    check += v;
    out[s] = v;
}

// The doublets transported forward along link d (family link included).
template <int ND, int HF, class S>
__device__ __forceinline__ void forward_doublets(const LevelPtrs<S>& L, int d, int c, Q<S> U, S th, Q<S> (&t)[ND])
{
    S sn, cs;
    gsincos(th, sn, cs);
#pragma unroll
    for (int db = 0; db < ND; db++) t[db] = transport(U, cs, sn, ld4<S>(L.ph[db], c));
    if constexpr (HF == kHfU1) {
        S hs, hc;
        gsincos(ld1<S>(L.hth[d], c), hs, hc);
        hf_act<HF>(t[0], t[1], hc, hs, Q<S>{(S)1, (S)0, (S)0, (S)0});
    } else if constexpr (HF == kHfSU2) {
        hf_act<HF>(t[0], t[1], (S)1, (S)0, ld4<S>(L.hq[d], c));
    }
}

template <class S, int MODEL, int HF, bool ENERGY>
__device__ __forceinline__ void link_role(const KConst<S>& F, const LevelPtrs<S>& now, const LevelPtrs<S>& past,
                                          const LinkSite& n, double (&e)[kRCount], unsigned& warn, S& check)
{
    using C = S;
    constexpr int ND = (MODEL == kModelSM) ? 1 : 2;
    const int d = n.d, c = n.c;
    const Q<C> Up = ld4<C>(past.q[d], c);
    const C tp = ld1<C>(past.th[d], c);
    const Q<C> U = ld4<C>(now.q[d], c);
    const C th = ld1<C>(now.th[d], c);
    C mag_e = (C)0, elec_e = (C)0, grad_e = (C)0, plaq2 = (C)0, plaq1 = (C)0;
    C M[3];
    link_force<ENERGY>(F, now.q, n, U, M, mag_e, plaq2, F.inv_g_sqr);
    C MY = phase_force<ENERGY>(F, now.th, n, th, mag_e, plaq1, F.inv_gp_sqr);
    Q<C> t[ND];
    forward_doublets<ND, HF>(now, d, c, U, th, t);
    C jh = (C)0;
#pragma unroll
    for (int db = 0; db < ND; db++) {
        const Q<C> u = t[db], f = ld4<C>(now.ph[db], c + n.pd);
        const C up = u.w * f.x - u.x * f.w, lo = u.y * f.z - u.z * f.y;
        MY += F.cY * (up + lo);
        M[0] += F.cI * (u.w * f.z - u.x * f.y + u.y * f.x - u.z * f.w);
        M[1] += F.cI * (-u.w * f.y - u.x * f.z + u.y * f.w + u.z * f.x);
        M[2] += F.cI * (up - lo);
        if (HF == kHfU1) jh += db ? -(up + lo) : up + lo;  // +theta_H on doublet 1, -theta_H on doublet 2
        if (ENERGY) {
            const C e0 = f.w - u.w, e1 = f.x - u.x, e2 = f.y - u.y, e3 = f.z - u.z;
            grad_e += F.e_grad[d] * (e0 * e0 + e1 * e1 + e2 * e2 + e3 * e3);
        }
    }
    advance_phase<ENERGY>(F, past.th[d], c, th, tp, MY, F.e_elec[d] * F.inv_gp_sqr, elec_e, warn, check);
    advance_link<ENERGY>(F, past.q[d], c, U, Up, M, F.e_elec[d] * F.inv_g_sqr, elec_e, warn, check);
    if constexpr (HF == kHfU1) {
        const C h = ld1<C>(now.hth[d], c);
        C none = (C)0;
        const C MH = phase_force<ENERGY>(F, now.hth, n, h, mag_e, none, F.inv_gpp_sqr) + F.cH * jh;
        advance_phase<ENERGY>(F, past.hth[d], c, h, ld1<C>(past.hth[d], c), MH, F.e_elec[d] * F.inv_gpp_sqr, elec_e,
                              warn, check);
    }
    if (ENERGY) {
        e[kRGrad] = (double)grad_e;
        e[kRMag] = (double)mag_e;
        e[kRElec] = (double)elec_e;
        e[kRPlaq2] = (double)plaq2;
        e[kRPlaq1] = (double)plaq1;
    }
}

// The family SU(2) link of direction d (WilsonLoops/Source/TwoHDM.cpp:484-551, 601-633, 702-745;
// currents Gradients/Source/TwoHDM.cpp:465-485).
template <class S, bool ENERGY>
__device__ __forceinline__ void family_role(const KConst<S>& F, const LevelPtrs<S>& now, const LevelPtrs<S>& past,
                                            const LinkSite& n, double (&e)[kRCount], unsigned& warn, S& check)
{
    using C = S;
    const int d = n.d, c = n.c;
    const Q<C> Hp = ld4<C>(past.hq[d], c);
    const Q<C> H = ld4<C>(now.hq[d], c);
    C mag_e = (C)0, elec_e = (C)0, none = (C)0;
    C M[3];
    link_force<ENERGY>(F, now.hq, n, H, M, mag_e, none, F.inv_gpp_sqr);
    Q<C> t[2];
    forward_doublets<2, kHfSU2>(now, d, c, ld4<C>(now.q[d], c), ld1<C>(now.th[d], c), t);
    const Q<C> f0 = ld4<C>(now.ph[0], c + n.pd), f1 = ld4<C>(now.ph[1], c + n.pd);
    const C t8[8] = {t[0].w, t[0].x, t[0].y, t[0].z, t[1].w, t[1].x, t[1].y, t[1].z};
    const C n8[8] = {f0.w, f0.x, f0.y, f0.z, f1.w, f1.x, f1.y, f1.z};
    C h4 = 0, h5 = 0, h6 = 0;
#pragma unroll
    for (int i = 0; i < 4; i += 2) {
        h4 += t8[i] * n8[i + 5] - t8[i + 1] * n8[i + 4] + t8[i + 4] * n8[i + 1] - t8[i + 5] * n8[i];
        h5 += -t8[i] * n8[i + 4] - t8[i + 1] * n8[i + 5] + t8[i + 4] * n8[i] + t8[i + 5] * n8[i + 1];
        h6 += t8[i] * n8[i + 1] - t8[i + 1] * n8[i] - t8[i + 4] * n8[i + 5] + t8[i + 5] * n8[i + 4];
    }
    M[0] += F.cH * h4;
    M[1] += F.cH * h5;
    M[2] += F.cH * h6;
    advance_link<ENERGY>(F, past.hq[d], c, H, Hp, M, F.e_elec[d] * F.inv_gpp_sqr, elec_e, warn, check);
    if (ENERGY) {
        e[kRMag] = (double)mag_e;
        e[kRElec] = (double)elec_e;
    }
}

template <class S, int MODEL, int HF, bool ENERGY>
__device__ __forceinline__ void doublet_role(const StepParams& P, const KConst<S>& F, const LevelPtrs<S>& now,
                                             const LevelPtrs<S>& past, int c, int x, int y, int z, double (&e)[kRCount],
                                             S& check)
{
    using C = S;
    constexpr int ND = (MODEL == kModelSM) ? 1 : 2;
    Q<C> fp[ND], fc[ND], D[ND];
#pragma unroll
    for (int db = 0; db < ND; db++) {
        fp[db] = ld4<C>(past.ph[db], c);
        fc[db] = ld4<C>(now.ph[db], c);
    }
    e[kRPot] = site_potential<MODEL, ENERGY>(P, F, fc, D);
#pragma unroll 1
    for (int a = 0; a < 3; a++) {
        int m, p;
        LinkSite::axis(P, a, x, y, z, m, p);
        const Q<C> U = ld4<C>(now.q[a], c), Um = ld4<C>(now.q[a], c + m);
        C sn, cs, sm, cm;
        gsincos(ld1<C>(now.th[a], c), sn, cs);
        gsincos(ld1<C>(now.th[a], c + m), sm, cm);
        Q<C> tm[ND], tp[ND];
#pragma unroll
        for (int db = 0; db < ND; db++) {
            tm[db] = transport(Um, cm, sm, ld4<C>(now.ph[db], c + m));
            tp[db] = transport_back(U, cs, sn, ld4<C>(now.ph[db], c + p));
        }
        if constexpr (HF == kHfU1) {
            C hs, hc, gs, gc;
            gsincos(ld1<C>(now.hth[a], c), hs, hc);
            gsincos(ld1<C>(now.hth[a], c + m), gs, gc);
            const Q<C> one = {(C)1, (C)0, (C)0, (C)0};
            hf_act<HF>(tm[0], tm[1], gc, gs, one);
            hf_act<HF>(tp[0], tp[1], hc, -hs, one);
        } else if constexpr (HF == kHfSU2) {
            hf_act<HF>(tm[0], tm[1], (C)1, (C)0, ld4<C>(now.hq[a], c + m));
            hf_act<HF>(tp[0], tp[1], (C)1, (C)0, qconj(ld4<C>(now.hq[a], c)));
        }
#pragma unroll
        for (int db = 0; db < ND; db++) {
            D[db] = qadd_scaled(D[db], F.ldt[a], tm[db]);
            D[db] = qadd_scaled(D[db], F.ldt[a], tp[db]);
        }
    }
    C kin_e = (C)0, phisq = (C)0;
#pragma unroll
    for (int db = 0; db < ND; db++)
        leapfrog_doublet<ENERGY>(F, fc[db], fp[db], D[db], past.ph[db], c, kin_e, phisq, check);
    if (ENERGY) {
        e[kRKin] = 0.5 * P.inv_sqr_dt * (double)kin_e;
        e[kRPhiSq] = (double)phisq;
    }
}

template <class S, int MODEL, int HF, bool ENERGY>
__global__ void __launch_bounds__(32 * role_count(HF)) role_step_kernel(const __grid_constant__ StepParams P,
                                                                       const __grid_constant__ KConst<S> F,
                                                                       const __grid_constant__ LevelPtrs<S> now,
                                                                       const __grid_constant__ LevelPtrs<S> past,
                                                                       unsigned* status, double* partials)
{
    constexpr int NR = role_count(HF);
    const int lane = threadIdx.x, role = threadIdx.y;
    const int c = blockIdx.x * 32 + lane;
    double e[kRCount];
#pragma unroll
    for (int k = 0; k < kRCount; k++) e[k] = 0.0;
    unsigned warn = 0;
    bool own = false;
    if (c < P.nsite) {
        const int r = c / P.nz, z = c - r * P.nz, x = r / P.ny, y = r - x * P.ny;
        own = counts(P, x);
        if (!frozen(P, x, y, z)) {  // Fixed faces: not evolved
            S check = (S)0;
            if (role < 3) {
                link_role<S, MODEL, HF, ENERGY>(F, now, past, LinkSite(P, c, role, x, y, z), e, warn, check);
            } else if (role == 3) {
                doublet_role<S, MODEL, HF, ENERGY>(P, F, now, past, c, x, y, z, e, check);
            } else {
                if constexpr (HF == kHfSU2)
                    family_role<S, ENERGY>(F, now, past, LinkSite(P, c, role - 4, x, y, z), e, warn, check);
            }
            if (!isfinite(check)) warn |= kWarnNonFinite;
        }
        if (!own) {  // ghost plane of an x-slab: no observables, no warnings
            warn = 0;
#pragma unroll
            for (int k = 0; k < kRCount; k++) e[k] = 0.0;
        }
    }
    if (ENERGY) {
        __shared__ double s_e[NR][kRCount][32];
        __shared__ double s_row[kRCount];
#pragma unroll
        for (int k = 0; k < kRCount; k++) s_e[role][k][lane] = e[k];
        __syncthreads();
        for (int k = role; k < kRCount; k += NR) {  // a slot per role: over the roles, then the sites
            double v = 0.0;
#pragma unroll
            for (int r = 0; r < NR; r++) v += s_e[r][k][lane];
            s_e[0][k][lane] = v;
            v = warp_sum(v);
            if (lane == 0) s_row[k] = v;
        }
        __syncthreads();
        if (role == 0) {
            if (P.loc_energy && own) {  // Energy's local densities (Analysers/Source/Energy.cpp:137-143)
                double t = 0.0;
                float* o = P.loc_energy + 6 * (size_t)c;
#pragma unroll
                for (int k = kRPot; k <= kRElec; k++) {
                    t += s_e[0][k][lane];
                    o[1 + k] = (float)s_e[0][k][lane];
                }
                o[0] = (float)t;
            }
            if (lane == 0) {
                double* row = partials + (size_t)blockIdx.x * kObsCount;
                row[kObsEnergy] = s_row[kRPot] + s_row[kRGrad] + s_row[kRKin] + s_row[kRMag] + s_row[kRElec];
                row[kObsPotential] = s_row[kRPot];
                row[kObsGradient] = s_row[kRGrad];
                row[kObsKinetic] = s_row[kRKin];
                row[kObsMagnetic] = s_row[kRMag];
                row[kObsElectric] = s_row[kRElec];
                row[kObsPlaqSU2] = s_row[kRPlaq2];
                row[kObsPlaqU1] = s_row[kRPlaq1];
                row[kObsPhiSq] = s_row[kRPhiSq];
            }
        }
    }
    if (warn) atomicOr(status, warn);
}

template <class S, int MODEL, int HF>
cudaError_t launch(const StepParams& P, const LevelPtrs<S>& now, const LevelPtrs<S>& past, unsigned* status,
                   double* partials, bool energy, cudaStream_t stream)
{
    const dim3 block(32, role_count(HF));
    const int grid = role_launch_blocks(P);
    if (energy)
        role_step_kernel<S, MODEL, HF, true><<<grid, block, 0, stream>>>(P, make_kconst<S>(P), now, past, status, partials);
    else
        role_step_kernel<S, MODEL, HF, false><<<grid, block, 0, stream>>>(P, make_kconst<S>(P), now, past, status, partials);
    return cudaGetLastError();
}

}  // namespace

int role_launch_blocks(const StepParams& P) { return (P.nsite + 31) / 32; }

template <class S, int MODEL>
cudaError_t launch_role_step(const StepParams& P, const LevelPtrs<S>& now, const LevelPtrs<S>& past, unsigned* status,
                             double* partials, bool energy, cudaStream_t stream)
{
    if constexpr (MODEL == kModel2HDM) {
        if (P.hf == kHfU1) return launch<S, MODEL, kHfU1>(P, now, past, status, partials, energy, stream);
        if (P.hf == kHfSU2) return launch<S, MODEL, kHfSU2>(P, now, past, status, partials, energy, stream);
    }
    return launch<S, MODEL, kHfNone>(P, now, past, status, partials, energy, stream);
}

#define GFT_INSTANTIATE_ROLE(S, M)                                                                            \
    template cudaError_t launch_role_step<S, M>(const StepParams&, const LevelPtrs<S>&, const LevelPtrs<S>&,  \
                                                unsigned*, double*, bool, cudaStream_t);
GFT_INSTANTIATE_ROLE(float, kModelSM)
GFT_INSTANTIATE_ROLE(float, kModel2HDM)
GFT_INSTANTIATE_ROLE(double, kModelSM)
GFT_INSTANTIATE_ROLE(double, kModel2HDM)

}  // namespace gft
