// gft_tiled_tile.cuh -- one tile of the TMA-staged step kernel, shared by the
// single-lattice kernel (gft_tiled_kernels.cu) and the persistent ensemble
// kernel (gft_ensemble.cu).
//
// A tile is a (TY x TZ) set of (y, z) columns of one lattice marching along x
// (the slowest-varying axis) over nloc planes.  The "now" level of every plane
// the stencil touches is brought into shared memory once, by the Tensor Memory
// Accelerator: one cp.async.bulk.tensor per field array per plane, a
// (TY+2) x (TZ+2) box including the one-site halo, completing on an mbarrier.
// The plane buffers form a ring: while plane x is computed from planes x and
// x+1 (what the site needs of plane x-1 it holds from its own last site, XCarry),
// the copy of plane x+2 is in flight.  Halo cells that wrap around
// the periodic boundary (tiles on the lattice faces) are outside the tensor
// and arrive zero-filled; the CTA overwrites them with plain loads of the
// wrapped sites.  The own-site past level is read and written directly
// (coalesced: consecutive threads are consecutive z).
//
// Bounded waits: every mbarrier wait gives up after 2 s of %globaltimer (or the
// shorter diagnostic limit StepParams::wait_limit_ns); the tile then waits, with
// the 2 s bound, for its copies still in flight, reports failure and the caller
// records kErrTimeout in the status word.
#pragma once

#include <cuda.h>

#include "gft_device.cuh"
#include "gft_launch.h"
#include "gft_shared_body.cuh"
#include "gft_step_body.cuh"

namespace gft {
namespace tiled {

constexpr unsigned kErrTimeout = 8u;

__device__ __forceinline__ unsigned smem_u32(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(unsigned long long* bar, unsigned count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_expect_tx(unsigned long long* bar, unsigned bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(unsigned long long* bar, unsigned parity)
{
    unsigned ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}

__device__ __forceinline__ unsigned long long globaltimer_ns()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Non-blocking test of phase `parity` of `bar`.
__device__ __forceinline__ bool mbar_test_wait(unsigned long long* bar, unsigned parity)
{
    unsigned ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}

constexpr unsigned long long kWaitLimitNs = 2000000000ull;  // 2 s

// Wait for phase `parity` of `bar`; false after `limit_ns` (0: 2 s).  A limit
// below 1 us is one non-blocking test (the diagnostic of gft_set_wait_limit:
// it fails whenever the copy has not landed yet).
__device__ __forceinline__ bool mbar_wait_bounded(unsigned long long* bar, unsigned parity, unsigned limit_ns = 0)
{
    if (limit_ns - 1u < 999u) return mbar_test_wait(bar, parity);  // 1 <= limit < 1 us
    if (mbar_try_wait(bar, parity)) return true;
    const unsigned long long t0 = globaltimer_ns();
    for (;;) {
        if (mbar_try_wait(bar, parity)) return true;
        if (globaltimer_ns() - t0 > (limit_ns ? (unsigned long long)limit_ns : kWaitLimitNs)) return false;
    }
}

__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* map, int c0, int c1, int c2,
                                            unsigned long long* bar)
{
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], "
        "[%5];" ::"r"(smem_u32(dst)),
        "l"(map), "r"(c0), "r"(c1), "r"(c2), "r"(smem_u32(bar))
        : "memory");
}

__device__ __forceinline__ void tma_prefetch_l2_3d(const CUtensorMap* map, int c0, int c1, int c2)
{
    asm volatile("cp.async.bulk.prefetch.tensor.3d.L2.global.tile [%0, {%1, %2, %3}];" ::"l"(map), "r"(c0), "r"(c1),
                 "r"(c2)
                 : "memory");
}

// Warm L2 with the own-site past-level tile of plane X (boxes without halo).
template <int ND>
__device__ __forceinline__ void prefetch_past(const TMaps& pm, int X, int y0, int z0)
{
#pragma unroll
    for (int d = 0; d < 3; d++) tma_prefetch_l2_3d(&pm.q[d], 4 * z0, y0, X);
#pragma unroll
    for (int d = 0; d < 3; d++) tma_prefetch_l2_3d(&pm.th[d], z0, y0, X);
#pragma unroll
    for (int k = 0; k < ND; k++) tma_prefetch_l2_3d(&pm.ph[k], 4 * z0, y0, X);
}

// Shared-memory plane geometry of a ring of NB planes: three (x, x + 1 and the one
// in flight), four for the bodies that also read plane x - 1.
template <class S, int TY, int TZ, int ND, int NB = 3>
struct Geom {
    static constexpr int TP = 16 / (int)sizeof(S);  // theta box starts TP columns left (16-byte aligned)
    static constexpr int ROWS = TY + 2;
    static constexpr int QP = TZ + 2;           // pitch of q / phi tiles (records of 4 S)
    static constexpr int HP = TZ + 2 * TP;      // pitch of theta tiles
    static constexpr int QBOX = ROWS * QP * 4 * (int)sizeof(S);
    static constexpr int HBOX = ROWS * HP * (int)sizeof(S);
    static constexpr int QB = (QBOX + 127) / 128 * 128;
    static constexpr int HB = (HBOX + 127) / 128 * 128;
    static constexpr int OFF_TH = 3 * QB;
    static constexpr int OFF_PH = 3 * QB + 3 * HB;
    static constexpr int BUF = 3 * QB + 3 * HB + ND * QB;
    static constexpr int NBUF = NB;
    static constexpr unsigned TX = 3 * QBOX + 3 * HBOX + ND * QBOX;  // bytes per plane copy
    static constexpr int SMEM = NBUF * BUF + 128 + 64;             // + alignment slack + barriers
};

// Staging area for the wrapped halo cells of one plane: one slot per halo cell (the halo_cell numbering), quaternion
// records [3 + ND][NH] then phases [3][NH], placed after the plane barriers.
// FP32 only (the tiled kernel serves the mixed form).
template <class S, int TY, int TZ, int ND, int NB = 3>
struct HaloStage {
    using G = Geom<S, TY, TZ, ND, NB>;
    static constexpr int NH = 2 * G::QP + 2 * TY;
    static constexpr int OFF_H = (3 + ND) * NH * 16;
    static constexpr int BYTES = OFF_H + 3 * NH * 4;
    static constexpr int OFFSET = G::NBUF * G::BUF + 64;  // 16-byte aligned (BUF is a multiple of 128)
    static constexpr int SMEM = OFFSET + BYTES + 128;      // + alignment slack of the dynamic base
    // Used only when it leaves the resident CTAs per SM unchanged: 228 KB of
    // shared memory per SM, 1 KB reserved and 16 bytes static per CTA, and on
    // logging steps the reduction's 32 rows of kObsCount doubles.
    static constexpr int per_sm(int dyn, bool energy)
    {
        return (228 * 1024) / (dyn + 16 + (energy ? 32 * kObsCount * 8 : 0) + 1024);
    }
    static constexpr bool use(bool energy)
    {
        return sizeof(S) == 4 && SMEM <= 227 * 1024 - 16 && per_sm(SMEM, energy) >= per_sm(G::SMEM, energy);
    }
    static constexpr bool kUse = use(false);
};

template <class S, int TY, int TZ, int ND>
struct TileAcc;

// Whether a tile's sites hand their loops and transports to one another (gft_shared_body.cuh).
// Not the float 2HDM's: with the hand-over buffers two CTAs fit an SM only over a ring of two
// planes, and two doublets' values do not fit 128 registers beside the energy's or the ensemble's
// list (us per step handed over / not: 192^3 plain 498 / 513, logging 737 / 665; 16 members of
// 64^3 361 / 346).
template <class S, int MODEL>
constexpr bool hands_over()
{
    return MODEL == kModelSM || sizeof(S) == 8;
}

// Plane buffers of the one-site tiles' ring (run_ring): three, or two where only they leave two
// CTAs per SM (the FP64 2HDM's, with its hand-over buffers).
template <class S, int MODEL>
constexpr int ring_planes()
{
    return MODEL != kModelSM && hands_over<S, MODEL>() ? 2 : 3;
}

// The buffers of the values handed from site to site within a tile (gft_shared_body.cuh), after
// the halo stage: for the y neighbours, slot y - y0 of the receiving row; for the
// z neighbours, the receiving row of the tile's first column.  Two planes of each: a plane's are
// read after its barrier, while faster warps write the next plane's.
template <class S, int MODEL, int TY, int TZ>
struct HandBuf {
    static constexpr int ND = (MODEL == kModelSM) ? 1 : 2;
    using H = HaloStage<S, TY, TZ, ND, ring_planes<S, MODEL>()>;
    using V = Handed<S, ND>;
    static constexpr int QUAD = 4 * (int)sizeof(S);
    static constexpr int YB = (2 + ND) * TY * TZ * QUAD, ZB = (2 + ND) * TY * QUAD;  // one plane's
    static constexpr int BYTES = 2 * (YB + ZB);
    static constexpr int OFFSET = (H::OFFSET + (sizeof(S) == 4 ? H::BYTES : 0) + 15) / 16 * 16;
    static constexpr int SMEM = OFFSET + BYTES + 128;  // + alignment slack of the dynamic base

    __device__ __forceinline__ static void put(unsigned char* b, int n, int i, const V& h)
    {
        S* p = reinterpret_cast<S*>(b);
        st4(p, i, h.fa[0], h.fa[1], h.fa[2], h.sa);
        st4(p, n + i, h.fb[0], h.fb[1], h.fb[2], h.sb);
#pragma unroll
        for (int db = 0; db < ND; db++) st4(p, (2 + db) * n + i, h.t[db].w, h.t[db].x, h.t[db].y, h.t[db].z);
    }
    __device__ __forceinline__ static V get(const unsigned char* b, int n, int i)
    {
        using A = TileAcc<S, TY, TZ, ND>;
        const Q<S> a = A::lds4(b, i), c = A::lds4(b, n + i);
        V h = {{a.w, a.x, a.y}, a.z, {c.w, c.x, c.y}, c.z, {}};
#pragma unroll
        for (int db = 0; db < ND; db++) h.t[db] = A::lds4(b, (2 + db) * n + i);
        return h;
    }
};

// Reference to a site in a staged plane: buffer base, q/phi cell, theta cell.
struct TRef {
    const unsigned char* b;
    int cq, ch;
};

template <class S, int TY, int TZ, int ND>
struct TileAcc {
    using G = Geom<S, TY, TZ, ND>;
    __device__ __forceinline__ Q<S> q(int d, TRef r) const { return lds4(r.b + d * G::QB, r.cq); }
    __device__ __forceinline__ S th(int d, TRef r) const
    {
        return reinterpret_cast<const S*>(r.b + G::OFF_TH + d * G::HB)[r.ch];
    }
    __device__ __forceinline__ Q<S> ph(int k, TRef r) const { return lds4(r.b + G::OFF_PH + k * G::QB, r.cq); }

    __device__ __forceinline__ static Q<S> lds4(const unsigned char* base, int cell)
    {
        if constexpr (sizeof(S) == 4) {
            const float4 v = reinterpret_cast<const float4*>(base)[cell];
            return {(S)v.x, (S)v.y, (S)v.z, (S)v.w};
        } else {
            const double2* p = reinterpret_cast<const double2*>(base) + 2 * cell;
            const double2 a = p[0], c = p[1];
            return {(S)a.x, (S)a.y, (S)c.x, (S)c.y};
        }
    }
};

template <class S, int TY, int TZ, int ND>
__device__ __forceinline__ void issue_plane(const TMaps& maps, unsigned char* buf, unsigned long long* bar, int X,
                                            int y0, int z0)
{
    using G = Geom<S, TY, TZ, ND>;
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    mbar_expect_tx(bar, G::TX);
#pragma unroll
    for (int d = 0; d < 3; d++) tma_load_3d(buf + d * G::QB, &maps.q[d], 4 * (z0 - 1), y0 - 1, X, bar);
#pragma unroll
    for (int d = 0; d < 3; d++) tma_load_3d(buf + G::OFF_TH + d * G::HB, &maps.th[d], z0 - G::TP, y0 - 1, X, bar);
#pragma unroll
    for (int k = 0; k < ND; k++) tma_load_3d(buf + G::OFF_PH + k * G::QB, &maps.ph[k], 4 * (z0 - 1), y0 - 1, X, bar);
}

// Halo cell handled by thread `tid` (2*QP + 2*TY cells: rows 0 and TY+1, then
// columns 0 and TZ+1); false if tid has none.
template <int TY, int QP>
__device__ __forceinline__ bool halo_cell(int tid, int& ly, int& lz)
{
    if (tid >= 2 * QP + 2 * TY) return false;
    if (tid < QP) {
        ly = 0;
        lz = tid;
    } else if (tid < 2 * QP) {
        ly = TY + 1;
        lz = tid - QP;
    } else if (tid < 2 * QP + TY) {
        ly = 1 + (tid - 2 * QP);
        lz = 0;
    } else {
        ly = 1 + (tid - 2 * QP - TY);
        lz = QP - 1;
    }
    return true;
}

// Warm L2 with the wrapped halo sites of plane X (one plane before they are
// patched), so the patch loads do not wait on DRAM.
template <class S, int TY, int TZ, int ND, class LV>
__device__ __forceinline__ void prefetch_wrapped_halo(const StepParams& P, const LV& now, int X, int y0,
                                                      int z0, int tid)
{
    using G = Geom<S, TY, TZ, ND>;
    int ly, lz;
    if (!halo_cell<TY, G::QP>(tid, ly, lz)) return;
    int y = y0 - 1 + ly, z = z0 - 1 + lz;
    if (y >= 0 && y < P.ny && z >= 0 && z < P.nz) return;
    y = (y < 0) ? y + P.ny : (y >= P.ny ? y - P.ny : y);
    z = (z < 0) ? z + P.nz : (z >= P.nz ? z - P.nz : z);
    const size_t s = ((size_t)X * P.ny + y) * P.nz + z;
#pragma unroll
    for (int d = 0; d < 3; d++) {
        asm volatile("prefetch.global.L2 [%0];" ::"l"(now.q[d] + 4 * s));
        asm volatile("prefetch.global.L2 [%0];" ::"l"(now.th[d] + s));
    }
#pragma unroll
    for (int k = 0; k < ND; k++) asm volatile("prefetch.global.L2 [%0];" ::"l"(now.ph[k] + 4 * s));
}

// Halo cells of plane X whose (y, z) leaves the lattice: load the wrapped
// site from global memory into the staged plane.
template <class S, int TY, int TZ, int ND, class LV>
__device__ __forceinline__ void patch_wrapped_halo(const StepParams& P, const LV& now, unsigned char* buf,
                                                   int X, int y0, int z0, int tid)
{
    using G = Geom<S, TY, TZ, ND>;
    int ly, lz;
    if (!halo_cell<TY, G::QP>(tid, ly, lz)) return;
    int y = y0 - 1 + ly, z = z0 - 1 + lz;
    if (y >= 0 && y < P.ny && z >= 0 && z < P.nz) return;  // delivered by the tensor copy
    y = (y < 0) ? y + P.ny : (y >= P.ny ? y - P.ny : y);
    z = (z < 0) ? z + P.nz : (z >= P.nz ? z - P.nz : z);
    const int s = (X * P.ny + y) * P.nz + z;
    const int cq = ly * G::QP + lz, ch = ly * G::HP + lz + G::TP - 1;
#pragma unroll
    for (int d = 0; d < 3; d++) {
        const Q<S> v = ld4<S>(now.q[d], s);
        st4(reinterpret_cast<S*>(buf + d * G::QB), cq, v.w, v.x, v.y, v.z);
        reinterpret_cast<S*>(buf + G::OFF_TH + d * G::HB)[ch] = ld1<S>(now.th[d], s);
    }
#pragma unroll
    for (int k = 0; k < ND; k++) {
        const Q<S> v = ld4<S>(now.ph[k], s);
        st4(reinterpret_cast<S*>(buf + G::OFF_PH + k * G::QB), cq, v.w, v.x, v.y, v.z);
    }
}

// As prefetch_wrapped_halo, but the wrapped sites of plane X go by cp.async
// into this thread's slots of the staging area, one plane before they are
// patched (patch_from_stage).
template <class S, int TY, int TZ, int ND, class LV>
__device__ __forceinline__ void stage_wrapped_halo(const StepParams& P, const LV& now, int X, int y0, int z0, int tid,
                                                   unsigned char* stage)
{
    using G = Geom<S, TY, TZ, ND>;
    using H = HaloStage<S, TY, TZ, ND>;
    static_assert(sizeof(S) == 4, "the halo stage holds FP32 records");
    int ly, lz;
    if (!halo_cell<TY, G::QP>(tid, ly, lz)) return;
    int y = y0 - 1 + ly, z = z0 - 1 + lz;
    if (y >= 0 && y < P.ny && z >= 0 && z < P.nz) return;
    y = (y < 0) ? y + P.ny : (y >= P.ny ? y - P.ny : y);
    z = (z < 0) ? z + P.nz : (z >= P.nz ? z - P.nz : z);
    const size_t s = ((size_t)X * P.ny + y) * P.nz + z;
#pragma unroll
    for (int d = 0; d < 3; d++) {
        cp_async16(stage + (d * H::NH + tid) * 16, now.q[d] + 4 * s);
        cp_async4(stage + H::OFF_H + (d * H::NH + tid) * 4, now.th[d] + s);
    }
#pragma unroll
    for (int k = 0; k < ND; k++) cp_async16(stage + ((3 + k) * H::NH + tid) * 16, now.ph[k] + 4 * s);
    cp_async_commit();
}

// The wrapped halo cells of the plane in `buf` from this thread's staging
// slots (filled by stage_wrapped_halo for that plane).
template <class S, int TY, int TZ, int ND>
__device__ __forceinline__ void patch_from_stage(const StepParams& P, unsigned char* buf, int y0, int z0, int tid,
                                                 const unsigned char* stage)
{
    using G = Geom<S, TY, TZ, ND>;
    using H = HaloStage<S, TY, TZ, ND>;
    int ly, lz;
    if (!halo_cell<TY, G::QP>(tid, ly, lz)) return;
    const int y = y0 - 1 + ly, z = z0 - 1 + lz;
    if (y >= 0 && y < P.ny && z >= 0 && z < P.nz) return;
    cp_async_wait_all();
    const int cq = ly * G::QP + lz, ch = ly * G::HP + lz + G::TP - 1;
    const float4* sq = reinterpret_cast<const float4*>(stage);
    const float* sh = reinterpret_cast<const float*>(stage + H::OFF_H);
#pragma unroll
    for (int d = 0; d < 3; d++) {
        reinterpret_cast<float4*>(buf + d * G::QB)[cq] = sq[d * H::NH + tid];
        reinterpret_cast<float*>(buf + G::OFF_TH + d * G::HB)[ch] = sh[d * H::NH + tid];
    }
#pragma unroll
    for (int k = 0; k < ND; k++) reinterpret_cast<float4*>(buf + G::OFF_PH + k * G::QB)[cq] = sq[(3 + k) * H::NH + tid];
}

// Parity of the completed phases of the plane barriers (bit b for
// barrier b), carried from tile to tile by a persistent CTA (every thread
// holds the same value).
struct RingPhase {
    unsigned bits;
};

// The plane ring of one tile (planes x0 .. x0+nloc-1 of columns y0.., z0..):
// TMA copies, waits, wrapped-halo patches and one CTA barrier per plane.
// body(i, bm, bc, bp) evolves the tile's sites of plane x0 + i from the staged
// planes bc (x) and bp (x + 1), and with NB = 4 also bm (x - 1); close(i) follows the
// plane's barrier and reads none of them.  With NB < 4,
// start(bc, bp) is called first, on the planes x0 - 1 and x0: what the first sites
// need of the plane before them.
// NB, the plane buffers: with 3 (or 4) the copy of a plane is in flight while the one
// before it is computed, and is waited for ahead of the barrier, which publishes its patches.
// With 2 it is issued into the buffer that the barrier frees and lands during close(i); it is
// waited for ahead of body, and a tile with wrapped halo cells takes a second barrier to publish them.
// tid: the thread's index in the CTA
// (the halo cells and the copy issue are divided by it).  smem: NBUF plane
// buffers followed by NBUF initialised mbarriers; s_abort: a shared flag that
// is 0 on entry.  Returns false (on every thread) if a wait gave up; the ring
// is then drained and must not be reused.  LV: the level pointer struct (its
// q / th / ph members are read).
// STAGE: the wrapped halo cells of a plane are copied by cp.async into
// `stage` (HaloStage) a plane ahead (NB = 2: with its copy), instead of prefetched into L2
// and loaded after the plane's wait.
template <class S, int TY, int TZ, int ND, class LV, bool STAGE, int NB, class Start, class Body, class Close>
__device__ __forceinline__ bool run_ring(const TMaps& maps, const TMaps& pmaps, const StepParams& P, const LV& now,
                                         int y0, int z0, int x0, int nloc, unsigned char* smem,
                                         unsigned long long* bars, RingPhase& ring, int* s_abort,
                                         unsigned char* stage, int tid, Start&& start, Body&& body,
                                         Close&& close)
{
    using G = Geom<S, TY, TZ, ND, NB>;
    constexpr bool BACK = NB == 4, LATE = NB == 2;
    // the plane whose buffer is free once plane i has been computed: i + FREE (relative planes)
    constexpr int FREE = BACK ? 0 : 1;
    const int nplanes = nloc + 2;  // planes x0-1 .. x0+nloc
    const bool wraps = (y0 == 0) || (y0 + TY == P.ny) || (z0 == 0) || (z0 + TZ == P.nz);
    auto plane_x = [&](int p) {  // global x of relative plane p (p = 0 is x0 - 1)
        int X = x0 - 1 + p;
        return (X < 0) ? X + P.nx : (X >= P.nx ? X - P.nx : X);
    };
    // buffer of relative plane p and the parity of its phase
    auto slot = [&](int p) { return p % G::NBUF; };
    auto parity = [&](int p) { return ((ring.bits >> slot(p)) ^ (unsigned)(p / G::NBUF)) & 1u; };
    auto issue = [&](int p) {
        issue_plane<S, TY, TZ, ND>(maps, smem + slot(p) * G::BUF, &bars[slot(p)], plane_x(p), y0, z0);
    };
    auto wait = [&](int p) { return mbar_wait_bounded(&bars[slot(p)], parity(p), P.wait_limit_ns); };
    auto halo_ahead = [&](int p) {
        if constexpr (STAGE)
            stage_wrapped_halo<S, TY, TZ, ND>(P, now, plane_x(p), y0, z0, tid, stage);
        else
            prefetch_wrapped_halo<S, TY, TZ, ND>(P, now, plane_x(p), y0, z0, tid);
    };
    auto patch = [&](int p) {
        if constexpr (STAGE)
            patch_from_stage<S, TY, TZ, ND>(P, smem + slot(p) * G::BUF, y0, z0, tid, stage);
        else
            patch_wrapped_halo<S, TY, TZ, ND>(P, now, smem + slot(p) * G::BUF, plane_x(p), y0, z0, tid);
    };

    constexpr int FIRST = LATE ? 2 : 3;  // planes resident and patched before the first body
    if (tid == 0) {
        for (int p = 0; p < min(G::NBUF, nplanes); p++) issue(p);
    }
    if (tid == 32 % (TY * TZ)) {
        // past level of the first two planes computed (relative planes 1 and 2)
        for (int p = 1; p <= 2 && p <= nloc; p++) prefetch_past<ND>(pmaps, plane_x(p), y0, z0);
    }
    if (wraps && FIRST < nplanes) halo_ahead(FIRST);

    bool ok = true;
    for (int p = 0; p < FIRST; p++) {  // nplanes >= 3
        ok = ok && wait(p);
        if (ok && wraps) patch_wrapped_halo<S, TY, TZ, ND>(P, now, smem + slot(p) * G::BUF, plane_x(p), y0, z0, tid);
    }
    if (!ok) *s_abort = 1;
    __syncthreads();
    // on a failed wait: the copies of planes [drain0, drain1) may still be in flight
    int drain0 = 0, drain1 = min(G::NBUF, nplanes);
    bool aborted = *s_abort != 0;

    if constexpr (!BACK) {
        if (!aborted) {
            start(smem, smem + G::BUF);
            __syncthreads();  // plane 0's buffer is free
            if (tid == 0 && G::NBUF < nplanes) issue(G::NBUF);
        }
    }

    for (int i = 0; i < nloc && !aborted; i++) {
        const int nxt = i + FREE + G::NBUF;  // the plane copied into the buffer freed by this one
        bool okn = true;
        if constexpr (LATE) {
            // plane i+2, issued after the last barrier
            okn = wait(i + 2);
            if (wraps) {
                if (okn) patch(i + 2);
                __syncthreads();
            }
            okn = __all_sync(0xffffffffu, okn);  // the body's shuffles need the whole warp
        }
        if (okn)
            body(i, smem + slot(i) * G::BUF, smem + slot(i + 1) * G::BUF, smem + slot(i + 2) * G::BUF);
        if constexpr (!LATE) {
            // plane i+3 (x+2) for the next site; its copy was issued one plane ago
            if (i + 3 < nplanes) {
                okn = wait(i + 3);
                if (okn && wraps) patch(i + 3);
            }
        }
        if (!okn) *s_abort = 1;
        __syncthreads();
        if (*s_abort) {  // the planes before these were waited for; the last copy issued was plane nxt-1
            aborted = true;
            drain0 = LATE ? i + 2 : i + 3;
            drain1 = min(nplanes, nxt);
            break;
        }
        if (tid == 32 % (TY * TZ) && i + 3 <= nloc) prefetch_past<ND>(pmaps, plane_x(i + 3), y0, z0);
        if (wraps && i + FIRST + 1 < nplanes) halo_ahead(i + FIRST + 1);
        if (tid == 0 && nxt < nplanes) issue(nxt);
        close(i);
    }
    if constexpr (STAGE) cp_async_wait_all();  // a staged plane not patched (abort) is still in flight
    if (aborted) {
        // drain: wait (bounded) for the copies still in flight into this CTA's buffers
        if (tid == 0)
            for (int p = drain0; p < drain1; p++) mbar_wait_bounded(&bars[slot(p)], parity(p));
        __syncthreads();
        return false;
    }
#pragma unroll
    for (int b = 0; b < G::NBUF; b++)
        if (b < nplanes) ring.bits ^= (((unsigned)((nplanes - b + G::NBUF - 1) / G::NBUF)) & 1u) << b;
    return true;
}

// Stencil references of the site in cell (cq0, ch0) of the staged planes bm, bc, bp.
template <int QP, int HP>
__device__ __forceinline__ Stencil<TRef> plane_stencil(const unsigned char* bm, const unsigned char* bc,
                                                       const unsigned char* bp, int cq0, int ch0)
{
    Stencil<TRef> n;
    n.c = {bc, cq0, ch0};
    n.m[0] = {bm, cq0, ch0};
    n.p[0] = {bp, cq0, ch0};
    n.m[1] = {bc, cq0 - QP, ch0 - HP};
    n.p[1] = {bc, cq0 + QP, ch0 + HP};
    n.m[2] = {bc, cq0 - 1, ch0 - 1};
    n.p[2] = {bc, cq0 + 1, ch0 + 1};
    n.d01 = {bp, cq0 - QP, ch0 - HP};
    n.d02 = {bp, cq0 - 1, ch0 - 1};
    n.d10 = {bm, cq0 + QP, ch0 + HP};
    n.d12 = {bc, cq0 + QP - 1, ch0 + HP - 1};
    n.d20 = {bm, cq0 + 1, ch0 + 1};
    n.d21 = {bc, cq0 - QP + 1, ch0 - HP + 1};
    return n;
}

// Whether a step stages its wrapped halo cells: HaloStage holds FP32 records, and the room for
// them is there beside the hand-over buffers.
template <class S, int MODEL, int TY, int TZ, bool ENERGY>
constexpr bool tile_stage()
{
    if constexpr (hands_over<S, MODEL>())
        return sizeof(S) == 4;
    else
        return HaloStage<S, TY, TZ, 2>::use(ENERGY);
}

// Evolves one tile by one step, one site per thread (threads TZ x TY).
template <class S, int MODEL, int TY, int TZ, bool ENERGY, class LV>
__device__ __forceinline__ bool run_tile(const TMaps& maps, const TMaps& pmaps, const StepParams& P, const KConst<S>& F,
                                         const LV& now, const LV& past, int y0, int z0, int x0,
                                         int nloc, unsigned char* smem, unsigned long long* bars, RingPhase& ring,
                                         int* s_abort, double (&obs)[kObsCount], unsigned& warn)
{
    constexpr int ND = (MODEL == kModelSM) ? 1 : 2, NB = ring_planes<S, MODEL>();
    constexpr bool STAGE = tile_stage<S, MODEL, TY, TZ, ENERGY>();
    using G = Geom<S, TY, TZ, ND, NB>;
    using Acc = TileAcc<S, TY, TZ, ND>;
    const int tz = threadIdx.x, ty = threadIdx.y;
    const int tid = ty * TZ + tz;
    // own cells
    const int cq0 = (ty + 1) * G::QP + (tz + 1);
    const int ch0 = (ty + 1) * G::HP + (tz + 1) + G::TP - 1;
    const int y = y0 + ty, z = z0 + tz;
    XCarry<S, ND> carry;
    // Fixed y and z faces freeze whole columns, Fixed x faces the ends of a march: such sites
    // hand over their loops and transports, and keep their own words
    const bool column_frozen = ((P.fixed_axes & 2) && (y == 0 || y == P.ny - 1)) ||
                               ((P.fixed_axes & 4) && (z == 0 || z == P.nz - 1));
    auto frozen_at = [&](int x) { return column_frozen || ((P.fixed_axes & 1) && (x == 0 || x == P.nx - 1)); };
    auto start = [&](const unsigned char* bc, const unsigned char* bp) {
        site_carry<S, ND>(Acc{}, plane_stencil<G::QP, G::HP>(bc, bc, bp, cq0, ch0), carry);
    };
    unsigned char* stage = smem + HaloStage<S, TY, TZ, ND, NB>::OFFSET;
    if constexpr (hands_over<S, MODEL>()) {
        using HB = HandBuf<S, MODEL, TY, TZ>;
        OpenSite<S, ND> o;
        PastValues<S, ND, LV, !ENERGY> pv = {{past, 0}};
        auto ybuf = [&](int i) { return smem + HB::OFFSET + (i & 1) * HB::YB; };
        auto zbuf = [&](int i) { return smem + HB::OFFSET + 2 * HB::YB + (i & 1) * HB::ZB; };
        constexpr int NW = TY * TZ / 32;  // warps of the tile
        return run_ring<S, TY, TZ, ND, LV, STAGE, NB>(
            maps, pmaps, P, now, y0, z0, x0, nloc, smem, bars, ring, s_abort, stage, tid, start,
            [&](int i, const unsigned char*, const unsigned char* bc, const unsigned char* bp) {
                {  // the halo row's and column's lanes, on warps that change with the plane
                    const int h = (((tid >> 5) + i) % NW) * 32 + (tid & 31);
                    if (h < TZ + TY) {
                        const bool row = h < TZ;
                        const int ly = row ? 0 : h - TZ + 1, lz = row ? h + 1 : 0;
                        const int cq = ly * G::QP + lz, ch = ly * G::HP + lz + G::TP - 1;
                        Handed<S, ND> hh;
                        halo_hand_over<S>(Acc{}, row ? 1 : 2, TRef{bc, cq, ch}, TRef{bp, cq, ch},
                                          TRef{bc, cq + G::QP, ch + G::HP}, TRef{bc, cq + 1, ch + 1}, hh);
                        if (row)
                            HB::put(ybuf(i), TY * TZ, h, hh);
                        else
                            HB::put(zbuf(i), TY, h - TZ, hh);
                    }
                }
                Handed<S, ND> hy, hz;
                site_open<S, MODEL, ENERGY>(P, F, Acc{}, plane_stencil<G::QP, G::HP>(bc, bc, bp, cq0, ch0), carry, o, hy,
                                            hz);
                if (ty + 1 < TY) HB::put(ybuf(i), TY * TZ, tid + TZ, hy);
                // the z neighbour's, from the lane below; the first column's come through shared memory
                const S lz = tz == 0 ? (S)0 : F.ldt[2];
                Handed<S, ND> hv;
                auto up = [](S v) { return __shfl_up_sync(0xffffffffu, v, 1, TZ < 32 ? TZ : 32); };
#pragma unroll
                for (int k = 0; k < 3; k++) {
                    hv.fa[k] = up(hz.fa[k]);
                    hv.fb[k] = up(hz.fb[k]);
                }
                hv.sa = up(hz.sa);
                hv.sb = up(hz.sb);
#pragma unroll
                for (int db = 0; db < ND; db++) hv.t[db] = {up(hz.t[db].w), up(hz.t[db].x), up(hz.t[db].y), up(hz.t[db].z)};
                receive(o, 0, 1, lz, hv);
                const int x = x0 + i;
                pv.at.s = (x * P.ny + y) * P.nz + z;
                // ahead of the barrier: its wait covers the loads' latency (two doublets of doubles have
                // no registers for them there)
                if (ND == 1 && !frozen_at(x)) pv.load();
            },
            [&](int i) {
                const int x = x0 + i;
                if (frozen_at(x)) return;
                if (ND == 2) pv.load();
                receive(o, 0, 2, F.ldt[1], HB::get(ybuf(i), TY * TZ, tid));
                if (tz == 0) receive(o, 0, 1, F.ldt[2], HB::get(zbuf(i), TY, ty));
                site_close<S, ENERGY>(P, F, o, pv, obs, warn, counts(P, x));
            });
    } else {
        return run_ring<S, TY, TZ, ND, LV, STAGE, NB>(
            maps, pmaps, P, now, y0, z0, x0, nloc, smem, bars, ring, s_abort, stage, tid, start,
            [&](int i, const unsigned char*, const unsigned char* bc, const unsigned char* bp) {
                const Stencil<TRef> n = plane_stencil<G::QP, G::HP>(bc, bc, bp, cq0, ch0);
                const int x = x0 + i;
                if (column_frozen) return;
                if (frozen_at(x))
                    site_carry<S, ND>(Acc{}, n, carry);  // not evolved; the next site needs its loops
                else
                    site_step<S, MODEL, ENERGY, kHfNone, true>(P, F, Acc{}, n,
                                                               PastSite<S, LV>{past, (x * P.ny + y) * P.nz + z}, carry,
                                                               obs, warn, counts(P, x));
            },
            [](int) {});
    }
}

// Dynamic shared memory of a one-site tile kernel.
template <class S, int MODEL, int TY, int TZ, bool ENERGY>
constexpr int tile_smem()
{
    if constexpr (hands_over<S, MODEL>()) {
        constexpr int b = HandBuf<S, MODEL, TY, TZ>::SMEM;
        static_assert(b <= 227 * 1024 - 16 - 32 * kObsCount * 8, "shared memory of a tile");
        return b;
    } else {
        return tile_stage<S, MODEL, TY, TZ, ENERGY>() ? HaloStage<S, TY, TZ, 2>::SMEM : Geom<S, TY, TZ, 2>::SMEM;
    }
}

// Resident CTAs per SM that shared memory admits, at most 512 threads: 228 KB per SM, 1 KB
// reserved per CTA, the logging steps' reduction rows.
template <class S, int MODEL, int TY, int TZ>
constexpr int tile_ctas()
{
    constexpr int plain = tile_smem<S, MODEL, TY, TZ, false>();
    constexpr int logging = tile_smem<S, MODEL, TY, TZ, true>() + 32 * kObsCount * 8;
    constexpr int smem = (plain > logging ? plain : logging) + 16 + 1024;
    constexpr int by_smem = (228 * 1024) / smem, by_threads = 512 / (TY * TZ);
    constexpr int b = by_smem < by_threads ? by_smem : by_threads;
    return b < 1 ? 1 : b;
}

}  // namespace tiled
}  // namespace gft
