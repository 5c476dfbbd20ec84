// gft_fast_kernels.cu -- throughput forms of the leapfrog step, one thread per
// site with neighbours read through L1/L2 (any lattice size), and the Gauss
// residual kernel.  The per-site arithmetic is gft_step_body.cuh.
//
//   GFT_FORM_FP64  : S = double.
//   GFT_FORM_MIXED : S = float (see gft_step_body.cuh for where precision is kept).
#include "gft_device.cuh"
#include "gft_launch.h"
#include "gft_math.cuh"
#include "gft_gauss_body.cuh"
#include "gft_step_body.cuh"

namespace gft {
namespace {

// Neighbour offsets: the site index is linear in (x, y, z), so the wrap of
// each axis contributes an independent offset.
struct Offs {
    int c, m[3], p[3];
};

__device__ __forceinline__ Offs offsets(const StepParams& P, int x, int y, int z)
{
    Offs o;
    const int plane = P.ny * P.nz;
    o.c = (x * P.ny + y) * P.nz + z;
    o.m[0] = (x == 0) ? (P.nx - 1) * plane : -plane;
    o.p[0] = (x + 1 == P.nx) ? -(P.nx - 1) * plane : plane;
    o.m[1] = (y == 0) ? (P.ny - 1) * P.nz : -P.nz;
    o.p[1] = (y + 1 == P.ny) ? -(P.ny - 1) * P.nz : P.nz;
    o.m[2] = (z == 0) ? P.nz - 1 : -1;
    o.p[2] = (z + 1 == P.nz) ? -(P.nz - 1) : 1;
    return o;
}

// Field access through L1/L2 (read-only path) for the "now" level.
template <class S>
struct GlobalAcc {
    LevelPtrs<S> L;
    __device__ __forceinline__ Q<S> q(int d, int s) const { return ld4<S>(L.q[d], s); }
    __device__ __forceinline__ S th(int d, int s) const { return ld1<S>(L.th[d], s); }
    __device__ __forceinline__ Q<S> ph(int k, int s) const { return ld4<S>(L.ph[k], s); }
    __device__ __forceinline__ S hth(int d, int s) const { return ld1<S>(L.hth[d], s); }
    __device__ __forceinline__ Q<S> hq(int d, int s) const { return ld4<S>(L.hq[d], s); }
};

constexpr int kStepThreads = 128;
constexpr int kGaussThreads = 256;  // 32 x 8: 2 % faster than 32 x 4 at 256^3 (624 against 638 us)

// The (z, y) patch of sites a block of T threads covers: bz x by of them, bz * by <= T, thread t at
// column t % bz, row t / bz.  32 x T/32 unless the shape that leaves the fewest threads without a site
// puts `gain` times as many to work (75 sites along z in three blocks of 32 idle a fifth of them).  Any
// other patch costs a run-time division and shorter or misaligned rows.  us per plain step of 600,000
// sites in the best shape / in 32 x 4, by how many times the threads with a site:
//   1.25 (nz = 75): SM mixed 45 / 53, 2HDM 59 / 63, FP64 SM 96 / 110; 1.47 (40): 47 / 64, 60 / 75, 102 / 129;
//   1.14 (130): 49 / 52, 61 / 62;  1.10 (84): 45 / 49, 60 / 58, FP64 SM 101 / 99;
//   1.04 (56): 47 / 49, 61 / 58, 107 / 99;  1.00 (60): 48 / 47, 61 / 55, 102 / 95.
// Logging steps hide the cost (84: 2HDM 74 / 81, FP64 193 / 203; 144, 1.07: 74 / 78, 188 / 195), and so does the
// family SU(2) (84: 93 / 95).  Up to two blocks of 32 x 4 per SM every block runs at once and a step takes
// one thread's time, which a patch only lengthens (18 x 32 x 40, 288 blocks: SM mixed 4.9 / 4.7, 2HDM 5.2 /
// 5.0, FP64 SM 8.2 / 7.3; 24 x 32 x 40, 384: 5.0 / 5.5, 5.2 / 5.8, 8.0 / 9.0).  The mixed Gauss pass runs faster in narrow rows at equal use (60: 21.4 /
// 22.5), the FP64 one slower (28.5 / 26.0).
struct Patch {
    int bz, by;
    int inv;  // t / bz = t * inv >> 16, exact for t < 1024 and bz <= 64
};

constexpr double kPatchGain = 1.03, kPatchGainPlain = 1.12;
template <class S, int MODEL, int HF>
constexpr double step_gain(bool energy)
{
    return energy || (sizeof(S) == 4 && (MODEL == kModelSM || HF != kHfNone)) ? kPatchGain : kPatchGainPlain;
}
constexpr double gauss_gain(bool fp32) { return fp32 ? 0.99 : 1.12; }

Patch pick_patch(const StepParams& P, int threads, double gain)
{
    const Patch rows = {32, threads / 32, 65536 / 32};
    if (P.nz % 32 == 0) return rows;
    if (threads == kStepThreads &&
        (long long)((P.nz + 31) / 32) * ((P.ny + rows.by - 1) / rows.by) * P.nx <= 2 * 148)
        return rows;
    auto used = [&](int bz, int by) {
        const double cover = (double)((P.nz + bz - 1) / bz) * ((P.ny + by - 1) / by) * threads;
        return (double)P.nz * P.ny / cover;
    };
    Patch best = rows;
    double most = 0.0;
    for (int bz = 8; bz <= 64; bz++) {
        const double u = used(bz, threads / bz);
        if (u > most * 1.02) {  // wider rows only where they pay
            most = u;
            best = {bz, threads / bz, (65536 + bz - 1) / bz};
        }
    }
    return most > gain * used(rows.bz, rows.by) ? best : rows;
}

dim3 patch_grid(const StepParams& P, const Patch& p)
{
    return dim3((P.nz + p.bz - 1) / p.bz, (P.ny + p.by - 1) / p.by, P.nx);
}

// The thread's site; false past the patch or the lattice.  ANY: any patch; else 32 x T/32, known
// to the compiler (the run-time division costs the FP64 2HDM step registers it has not: 1272
// against 1160 us at 192^3).
template <int T, bool ANY>
__device__ __forceinline__ bool patch_site(const StepParams& P, const Patch& p, int& x, int& y, int& z)
{
    x = blockIdx.z;
    if constexpr (ANY) {
        const int ty = (int)(threadIdx.x * p.inv) >> 16, tz = (int)threadIdx.x - ty * p.bz;
        z = blockIdx.x * p.bz + tz;
        y = blockIdx.y * p.by + ty;
        return ty < p.by && z < P.nz && y < P.ny;
    } else {
        z = blockIdx.x * 32 + (threadIdx.x & 31);
        y = blockIdx.y * (T / 32) + (threadIdx.x >> 5);
        return z < P.nz && y < P.ny;
    }
}

// One thread per site; the kernel below instantiates it with its launch bounds.
template <class S, int MODEL, int HF, bool ENERGY, bool ANY>
__device__ __forceinline__ void fast_step_body(StepParams P, KConst<S> F, LevelPtrs<S> now,
                                               LevelPtrs<S> past, Patch p, unsigned* status,
                                               double* partials)
{
    int x, y, z;
    const bool in = patch_site<kStepThreads, ANY>(P, p, x, y, z);
    double obs[kObsCount];
#pragma unroll
    for (int k = 0; k < kObsCount; k++) obs[k] = 0.0;
    unsigned warn = 0;
    if (in && !frozen(P, x, y, z)) {  // Fixed faces: not evolved
        const Offs o = offsets(P, x, y, z);
        Stencil<int> n;
        n.c = o.c;
#pragma unroll
        for (int a = 0; a < 3; a++) {
            n.m[a] = o.c + o.m[a];
            n.p[a] = o.c + o.p[a];
        }
        n.d01 = o.c + o.p[0] + o.m[1];
        n.d02 = o.c + o.p[0] + o.m[2];
        n.d10 = o.c + o.p[1] + o.m[0];
        n.d12 = o.c + o.p[1] + o.m[2];
        n.d20 = o.c + o.p[2] + o.m[0];
        n.d21 = o.c + o.p[2] + o.m[1];
        XCarry<S, (MODEL == kModelSM) ? 1 : 2> carry;  // of a march; not read here
        site_step<S, MODEL, ENERGY, HF>(P, F, GlobalAcc<S>{now}, n, PastSite<S>{past, o.c}, carry, obs, warn,
                                        counts(P, x));
    }
    if (ENERGY) {
        energy_total(obs);
        const int b = blockIdx.x + gridDim.x * (blockIdx.y + gridDim.y * blockIdx.z);
        block_reduce_store<kObsCount>(obs, partials + (size_t)b * kObsCount, kObsCount);
    }
    if (warn) atomicOr(status, warn);
}

// Resident blocks per SM the launch bounds of an instance ask for: as many as its
// registers take with no or a few spilled words, since the warps hide the
// neighbour loads' latency (us per step on a B200, unbounded / bounded):
//   FP64 SM 256^3: three blocks (168 registers) 2926 / 2267, logging 3499 / 3471; four spill, and
//     measured 2146 and 3228 last (5 % slower than three when the bound was set);
//   FP64 2HDM: two blocks (254 registers), as without a bound;
//   float 2HDM 192^3: four blocks (128) 646 / 545, logging 756 / 748;
//   float 2HDM with the family SU(2) 96 x 96 x 192: three blocks (168) 305 / 235, logging 340 / 340;
//   float SM: 86-100 registers, five blocks either way.
template <class S, int MODEL, int HF>
constexpr int fast_min_blocks()
{
    if (sizeof(S) == 8) return MODEL == kModelSM ? 3 : 2;
    if (MODEL == kModelSM) return 5;
    return HF == kHfSU2 ? 3 : 4;
}

template <class S, int MODEL, int HF, bool ENERGY, bool ANY>
__global__ void __launch_bounds__(kStepThreads, fast_min_blocks<S, MODEL, HF>())
    fast_step_kernel(StepParams P, KConst<S> F, LevelPtrs<S> now, LevelPtrs<S> past, Patch p, unsigned* status,
                     double* partials)
{
    fast_step_body<S, MODEL, HF, ENERGY, ANY>(P, F, now, past, p, status, partials);
}

// Gauss-law residual after a step (gauss_site in gft_step_body.cuh), one
// thread per site: every load of a site is independent of the others, which
// keeps the most loads in flight (a march along x that carries the x - 1 links
// in registers serialises them and measured slower).
template <class S, int MODEL, int HF, bool ANY>
__global__ void __launch_bounds__(kGaussThreads) fast_gauss_kernel(StepParams P, LevelPtrs<S> now, LevelPtrs<S> fut, Patch p,
                                                         double* partials)
{
    constexpr int NG = 2 * hf_neq(HF);
    int x, y, z;
    const bool in = patch_site<kGaussThreads, ANY>(P, p, x, y, z);
    double v[NG];
#pragma unroll
    for (int k = 0; k < NG; k++) v[k] = 0.0;
    if (in && counts(P, x) && !frozen(P, x, y, z)) {
        const Offs o = offsets(P, x, y, z);
        gauss_site<S, MODEL, HF>(P, now, fut, o.c, o.c + o.m[0], o.c + o.m[1], o.c + o.m[2], v);
    }
    const int blk = blockIdx.x + gridDim.x * (blockIdx.y + gridDim.y * blockIdx.z);
    block_reduce_store<NG>(v, partials + (size_t)blk * NG, NG / 2);
}

// The same over 7 x 32 tiles marching along x, the FP32 fields' links once each
// (gft_gauss_body.cuh).  Two blocks per SM, each an equal share of all tiles' planes.
constexpr int kGaussCtas = 2 * 148;

template <int MODEL>
__global__ void __launch_bounds__(kGaussTileThreads, 2)
    gauss_tile_kernel(StepParams P, LevelPtrs<float> now, LevelPtrs<float> fut, double* partials)
{
    __shared__ GaussBuf sm;
    double v[kGaussSlots];
#pragma unroll
    for (int k = 0; k < kGaussSlots; k++) v[k] = 0.0;
    const long long w = gauss_tile_planes(P);
    gauss_planes<MODEL>(P, now, fut, (int)(w * blockIdx.x / gridDim.x), (int)(w * (blockIdx.x + 1) / gridDim.x), sm, v);
    block_reduce_store<kGaussSlots>(v, partials + (size_t)blockIdx.x * kGaussSlots, 4);
}

template <class S, int MODEL, int HF>
void fast_step_launch(const StepParams& P, const LevelPtrs<S>& now, const LevelPtrs<S>& past, unsigned* status,
                      double* partials, bool energy, cudaStream_t stream)
{
    const Patch p = pick_patch(P, kStepThreads, step_gain<S, MODEL, HF>(energy));
    const bool any = p.bz != 32;
    auto k = energy ? (any ? fast_step_kernel<S, MODEL, HF, true, true> : fast_step_kernel<S, MODEL, HF, true, false>)
                    : (any ? fast_step_kernel<S, MODEL, HF, false, true> : fast_step_kernel<S, MODEL, HF, false, false>);
    k<<<patch_grid(P, p), kStepThreads, 0, stream>>>(P, make_kconst<S>(P), now, past, p, status, partials);
}

template <class S, int MODEL, int HF>
void fast_gauss_launch(const StepParams& P, const LevelPtrs<S>& now, const LevelPtrs<S>& fut, double* partials,
                       cudaStream_t stream)
{
    const Patch p = pick_patch(P, kGaussThreads, gauss_gain(sizeof(S) == 4));
    auto k = p.bz != 32 ? fast_gauss_kernel<S, MODEL, HF, true> : fast_gauss_kernel<S, MODEL, HF, false>;
    k<<<patch_grid(P, p), kGaussThreads, 0, stream>>>(P, now, fut, p, partials);
}

}  // namespace

static int patch_blocks(const StepParams& P, int threads, double gain)
{
    const dim3 g = patch_grid(P, pick_patch(P, threads, gain));
    return (int)(g.x * g.y * g.z);
}

// Small lattices divide a site's update over several warps (gft_role_kernels.cu): up to about one
// warp of sites per scheduler (592 of them), where one thread per site leaves them waiting on one
// chain of instructions each.  us per step replayed from a graph, divided / one thread per site:
//   16^3: SM mixed 2.9 / 3.9, FP64 3.7 / 6.1, 2HDM with the family SU(2) 3.3 / 6.1, FP64 4.1 / 8.9
//   24^3:          3.6 / 4.2,      4.7 / 5.9,                            4.7 / 6.7,      8.2 / 8.9
//   32^3:          5.0 / 4.7,      8.7 / 7.0,                            9.3 / 6.9,       17 / 12
constexpr int kRoleMaxSites = 16384;
static bool use_roles(const StepParams& P) { return P.nsite <= kRoleMaxSites; }

int fast_launch_blocks(const StepParams& P, bool divide)
{
    return divide && use_roles(P) ? role_launch_blocks(P) : patch_blocks(P, kStepThreads, kPatchGain);
}

// The mixed form's Gauss pass runs in tiles from 300,000 sites on (its 296 blocks then march four
// planes at least, each after one more) where at most a third of the tiles' sites lie past a ragged
// edge.  us per pass with its reduction, tiles / one thread per site: SM 48^3 17 / 15, 64^3 21 / 21,
// 100^3 46 / 63, 150 x 100 x 75 51 / 67, 128^3 72 / 101, 256^3 467 / 723; 2HDM 64^3 22 / 21, 96^3 49 / 56,
// 192^3 264 / 293.  The FP64 form's words would not fit the registers; it keeps one thread per site.
constexpr int kGaussTileSites = 300000;
static bool gauss_in_tiles(const StepParams& P, bool fp32)
{
    const double padded = (double)gauss_tile_planes(P) * kGaussTileY * kGaussTileZ;
    return fp32 && P.hf == kHfNone && P.nsite >= kGaussTileSites && padded <= 1.5 * P.nsite;
}

int fast_gauss_blocks(const StepParams& P, bool fp32)
{
    return gauss_in_tiles(P, fp32) ? kGaussCtas : patch_blocks(P, kGaussThreads, gauss_gain(fp32));
}

// P.hf selects the Higgs-family variant (2HDM only); the Gauss kernel writes
// 2 * gaugeNum partial slots per block.
template <class S, int MODEL>
cudaError_t launch_fast_step(const StepParams& P, const LevelPtrs<S>& now, const LevelPtrs<S>& past, unsigned* status,
                             double* partials, bool energy, bool divide, cudaStream_t stream)
{
    if (divide && use_roles(P)) return launch_role_step<S, MODEL>(P, now, past, status, partials, energy, stream);
    if constexpr (MODEL == kModel2HDM) {
        if (P.hf == kHfU1)
            fast_step_launch<S, MODEL, kHfU1>(P, now, past, status, partials, energy, stream);
        else if (P.hf == kHfSU2)
            fast_step_launch<S, MODEL, kHfSU2>(P, now, past, status, partials, energy, stream);
        else
            fast_step_launch<S, MODEL, kHfNone>(P, now, past, status, partials, energy, stream);
    } else {
        fast_step_launch<S, MODEL, kHfNone>(P, now, past, status, partials, energy, stream);
    }
    return cudaGetLastError();
}

template <class S, int MODEL>
cudaError_t launch_fast_gauss(const StepParams& P, const LevelPtrs<S>& now, const LevelPtrs<S>& fut, double* partials,
                              cudaStream_t stream)
{
    if constexpr (sizeof(S) == 4) {
        if (gauss_in_tiles(P, true)) {
            gauss_tile_kernel<MODEL><<<kGaussCtas, kGaussTileThreads, 0, stream>>>(P, now, fut, partials);
            return cudaGetLastError();
        }
    }
    if constexpr (MODEL == kModel2HDM) {
        if (P.hf == kHfU1)
            fast_gauss_launch<S, MODEL, kHfU1>(P, now, fut, partials, stream);
        else if (P.hf == kHfSU2)
            fast_gauss_launch<S, MODEL, kHfSU2>(P, now, fut, partials, stream);
        else
            fast_gauss_launch<S, MODEL, kHfNone>(P, now, fut, partials, stream);
    } else {
        fast_gauss_launch<S, MODEL, kHfNone>(P, now, fut, partials, stream);
    }
    return cudaGetLastError();
}

#define GFT_INSTANTIATE_FAST(S, M)                                                                                   \
    template cudaError_t launch_fast_step<S, M>(const StepParams&, const LevelPtrs<S>&, const LevelPtrs<S>&,         \
                                                unsigned*, double*, bool, bool, cudaStream_t);                        \
    template cudaError_t launch_fast_gauss<S, M>(const StepParams&, const LevelPtrs<S>&, const LevelPtrs<S>&,        \
                                                 double*, cudaStream_t);
GFT_INSTANTIATE_FAST(float, kModelSM)
GFT_INSTANTIATE_FAST(float, kModel2HDM)
GFT_INSTANTIATE_FAST(double, kModelSM)
GFT_INSTANTIATE_FAST(double, kModel2HDM)

}  // namespace gft
