// gft_gauss_body.cuh -- the Gauss-law residuals of a tile of FP32 fields, every link once.
//
// A site needs, of each of its three links and of each of its back neighbours' links, the
// vector of U_now^dag U_fut (or U_fut U_now^dag) and the sine of the phase's change.  One thread
// per site reads and converts six links; here a site works out its own three, hands them on --
// to its +x neighbour in its own registers (threads march along x), to +y through shared
// memory, to +z by shuffle -- and the eighth warp of a 7 x 32 tile supplies the row y0 - 1 and the
// column z0 - 1.  The next plane's words are loaded while this one's are worked on.
//
// The pass was bound by FP64 work: conversions of the FP32 words and the products.  Per site 38
// words (46 with two doublets) are converted instead of 68 (76), three sines taken instead of six; at SM
// 256^3 it reads at 5.4 TB/s (each word of both levels once) and takes 467 us with its reduction, 723
// one thread per site.  Two blocks of eight warps per SM have 128 registers, enough to hold the next plane of one
// doublet; two doublets' next plane is loaded at the end of a plane (2HDM 192^3 264 us; held it took 8 % longer).
// A block of 8 x 32 sites and a ninth warp leaves 96 registers and spills (870 us).
#pragma once

#include "gft_step_body.cuh"

namespace gft {

// What one link's change between the levels is to a constraint: the sine of its phase's change
// and the vector of U_now^dag U_fut (own site) or U_fut U_now^dag (the site ahead).
struct GaussTerm {
    double v[4];
};

// The terms of the link (now, fut, tnow, tfut) for its own site and for the site ahead.
__device__ __forceinline__ void gauss_terms(float4 n4, float4 f4, float tnow, float tfut, GaussTerm& own, GaussTerm& ahead)
{
    const Q<double> n = {n4.x, n4.y, n4.z, n4.w}, f = {f4.x, f4.y, f4.z, f4.w};
    own.v[0] = ahead.v[0] = gsin((double)tfut - (double)tnow);
    qmul_vec(qconj(n), f, own.v[1], own.v[2], own.v[3]);
    qmul_vec(f, qconj(n), ahead.v[1], ahead.v[2], ahead.v[3]);
}

// Words of one site and both levels.  The lanes of the halo warp hold links 1 and 2 of two
// different sites.
template <int ND>
struct GaussWords {
    float4 n[3], f[3], pn[ND], pf[ND];
    float tn[3], tf[3];
};

constexpr int kGaussTileY = 7, kGaussTileZ = 32, kGaussTileThreads = (kGaussTileY + 1) * kGaussTileZ;

// Shared memory: the y neighbours' values and the first column's z neighbours', a double per
// slot and component, two planes of each.
struct GaussBuf {
    double y[2][4][kGaussTileY * kGaussTileZ], z[2][4][kGaussTileY];
};

// Planes of tiles of a lattice, tile by tile: the work that blocks share out.
__host__ __device__ inline int gauss_tile_planes(const StepParams& P)
{
    return ((P.ny + kGaussTileY - 1) / kGaussTileY) * ((P.nz + kGaussTileZ - 1) / kGaussTileZ) * P.nx;
}

// Adds |violation| of the four constraints over the sites of the planes [w0, w1) of
// gauss_tile_planes to v[0..3] and takes their maxima into v[4..7].  Threads: a tile's sites and a
// halo warp.  Columns past the lattice's edges (a ragged edge) hand on what nobody takes and are
// not counted.
template <int MODEL, class LV>
__device__ __forceinline__ void gauss_planes(const StepParams& P, const LV& now, const LV& fut, int w0, int w1,
                                             GaussBuf& sm, double (&v)[kGaussSlots])
{
    constexpr int ND = (MODEL == kModelSM) ? 1 : 2, TY = kGaussTileY, TZ = kGaussTileZ;
    constexpr bool AHEAD = ND == 1;  // two doublets' words do not fit the registers twice
    const int tid = threadIdx.x, lane = tid & 31, ty = tid >> 5;
    const bool halo = ty == TY;
    const int plane = P.ny * P.nz, tiles_z = (P.nz + TZ - 1) / TZ;

    // of the plane whose words are loaded: its x, the sites within it of this thread's links (its
    // own, or the halo row's and column's) and whether its site counts but for x
    int x, s1, s2;
    bool in;
    auto place = [&](int w) {
        const int t = w / P.nx, y0 = (t / tiles_z) * TY, z0 = (t % tiles_z) * TZ;
        auto wrapped = [](int i, int n) { return i < 0 ? i + n : (i < n ? i : n - 1); };
        x = w - t * P.nx;
        const int y = y0 + ty, z = z0 + lane;
        s1 = wrapped(halo ? y0 - 1 : y, P.ny) * P.nz + wrapped(z, P.nz);
        s2 = halo ? wrapped(y0 + (lane < TY ? lane : 0), P.ny) * P.nz + wrapped(z0 - 1, P.nz) : s1;
        in = !halo && y < P.ny && z < P.nz && !((P.fixed_axes & 2) && (y == 0 || y == P.ny - 1)) &&
             !((P.fixed_axes & 4) && (z == 0 || z == P.nz - 1));
    };
    auto ld = [](const auto* p, int s) { return reinterpret_cast<const float4*>(p)[s]; };
    auto load_doublets = [&](GaussWords<ND>& w, int a) {
        if (halo) return;
#pragma unroll
        for (int k = 0; k < ND; k++) {
            w.pn[k] = ld(now.ph[k], a);
            w.pf[k] = ld(fut.ph[k], a);
        }
    };
    auto load = [&](GaussWords<ND>& w) {
        const int a = x * plane + s1, b = x * plane + s2;
        w.n[1] = ld(now.q[1], a);
        w.f[1] = ld(fut.q[1], a);
        w.tn[1] = now.th[1][a];
        w.tf[1] = fut.th[1][a];
        w.n[2] = ld(now.q[2], b);
        w.f[2] = ld(fut.q[2], b);
        w.tn[2] = now.th[2][b];
        w.tf[2] = fut.th[2][b];
        if (!halo) {
            w.n[0] = ld(now.q[0], a);
            w.f[0] = ld(fut.q[0], a);
            w.tn[0] = now.th[0][a];
            w.tf[0] = fut.th[0][a];
        }
        load_doublets(w, a);
    };
    auto put = [](auto& b, int i, const GaussTerm& t) {
#pragma unroll
        for (int k = 0; k < 4; k++) b[k][i] = t.v[k];
    };

    GaussTerm back = {};  // of the site before in the march
    GaussWords<ND> cur;
    place(w0);
    load(cur);
#pragma unroll 1
    for (int w = w0; w < w1; w++) {
        const int xc = x, c = x * plane + s1, par = w & 1;
        const bool count = in && counts(P, x) && !((P.fixed_axes & 1) && (x == 0 || x == P.nx - 1));
        if ((w == w0 || xc == 0) && !halo) {  // a march begins
            const int a = c + (xc == 0 ? (P.nx - 1) * plane : -plane);
            GaussTerm own;
            gauss_terms(ld(now.q[0], a), ld(fut.q[0], a), now.th[0][a], fut.th[0][a], own, back);
        }
        GaussWords<ND> next;
        if (AHEAD && w + 1 < w1) {
            if (++x == P.nx) place(w + 1);
            load(next);
        }

        GaussTerm e1, e2, ay, az;
        gauss_terms(cur.n[1], cur.f[1], cur.tn[1], cur.tf[1], e1, ay);
        if (ty + 1 != TY) put(sm.y[par], halo ? lane : tid + TZ, ay);
        gauss_terms(cur.n[2], cur.f[2], cur.tn[2], cur.tf[2], e2, az);
        if (halo && lane < TY) put(sm.z[par], lane, az);
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const double up = __shfl_up_sync(0xffffffffu, az.v[k], 1);
            if (lane != 0) e2.v[k] -= up;
        }
        __syncthreads();
        if (!halo) {
            GaussTerm e0, ax;
            gauss_terms(cur.n[0], cur.f[0], cur.tn[0], cur.tf[0], e0, ax);
            double el[4], gr[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
            for (int k = 0; k < 4; k++) {
                if (lane == 0) e2.v[k] -= sm.z[par][k][ty];
                el[k] = (e0.v[k] - back.v[k]) * P.lap[0];
                el[k] += (e1.v[k] - sm.y[par][k][tid]) * P.lap[1];
                el[k] += e2.v[k] * P.lap[2];
            }
            back = ax;
#pragma unroll
            for (int db = 0; db < ND; db++) {
                const Q<double> p = {cur.pn[db].x, cur.pn[db].y, cur.pn[db].z, cur.pn[db].w};
                const Q<double> q = {cur.pf[db].x, cur.pf[db].y, cur.pf[db].z, cur.pf[db].w};
                gr[0] += 0.25 * (p.w * q.x - p.x * q.w + p.y * q.z - p.z * q.y);
                gr[1] += 0.25 * (p.w * q.z - p.x * q.y + p.y * q.x - p.z * q.w);
                gr[2] += 0.25 * (-p.w * q.y - p.x * q.z + p.y * q.w + p.z * q.x);
                gr[3] += 0.25 * (p.w * q.x - p.x * q.w - p.y * q.z + p.z * q.y);
            }
            if (count) {
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    const double viol = el[k] - P.gsq[k] * gr[k], av = fabs(viol);
                    v[k] += av;
                    v[4 + k] = fmax(v[4 + k], av);
                    if (P.loc_gauss) P.loc_gauss[4 * (size_t)c + k] = (float)viol;  // GaugeCondition local violation
                }
            }
        }
        if (AHEAD) {
            cur = next;
        } else if (w + 1 < w1) {
            if (++x == P.nx) place(w + 1);
            load(cur);
        }
    }
}

}  // namespace gft
