// gft_reduce.cuh -- deterministic FP64 reduction of per-block partial rows.
#pragma once

#include <cuda_runtime.h>

namespace gft {

constexpr int kFinThreads = 1024;
constexpr int kMaxSlots = 16;

// One Neumaier-compensated addition: sum + comp is the running total.
__device__ __forceinline__ void add_compensated(double& sum, double& comp, double v)
{
    const double t = sum + v;
    comp += (fabs(sum) >= fabs(v)) ? (sum - t) + v : (v - t) + sum;
    sum = t;
}

// Reduces rows [b0, b1) of partials[*][nslots] over the whole block (blockDim.x
// = kFinThreads, 1-D), slot k with Neumaier compensation (k < max_from) or as a
// maximum (k >= max_from; values are >= 0).  A thread accumulates one slot, of
// every (kFinThreads / nslots)-th row, reading consecutive words with its
// neighbours; then warp k combines the threads of slot k.  The order is fixed, so
// the result is deterministic.  Thread k < nslots returns the total of slot k.
// The block is one chain of latencies: whole rows per thread, each thread holding
// sixteen pairs of accumulators, took 14 to 18 us for some hundreds of rows.
__device__ __forceinline__ double reduce_rows_block(const double* __restrict__ partials, int b0, int b1, int nslots,
                                                    int max_from)
{
    __shared__ double s_sum[kFinThreads];
    __shared__ double s_cmp[kFinThreads];
    __shared__ double s_out[kMaxSlots];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int groups = kFinThreads / nslots, used = groups * nslots;
    {
        double sum = 0.0, comp = 0.0;
        if (tid < used) {
            const bool is_max = tid % nslots >= max_from;
            const double* p = partials + (size_t)b0 * nslots;
            const int n = (b1 - b0) * nslots;
            int i = tid;
            for (; i + 3 * used < n; i += 4 * used) {  // four loads in flight
                const double v[4] = {p[i], p[i + used], p[i + 2 * used], p[i + 3 * used]};
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    if (is_max)
                        sum = fmax(sum, v[k]);
                    else
                        add_compensated(sum, comp, v[k]);
                }
            }
            for (; i < n; i += used) {
                if (is_max)
                    sum = fmax(sum, p[i]);
                else
                    add_compensated(sum, comp, p[i]);
            }
        }
        s_sum[tid] = sum;
        s_cmp[tid] = comp;
    }
    __syncthreads();
    if (warp < nslots) {
        const bool is_max = warp >= max_from;
        double sum = 0.0, comp = 0.0;
        for (int g = lane; g < groups; g += 32) {
            const double v = s_sum[g * nslots + warp];
            if (is_max) {
                sum = fmax(sum, v);
            } else {
                add_compensated(sum, comp, v);
                comp += s_cmp[g * nslots + warp];
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {  // a fixed tree
            const double v = __shfl_xor_sync(0xffffffffu, sum, o);
            const double c = __shfl_xor_sync(0xffffffffu, comp, o);
            if (is_max) {
                sum = fmax(sum, v);
            } else {
                add_compensated(sum, comp, v);
                comp += c;
            }
        }
        if (lane == 0) s_out[warp] = is_max ? sum : sum + comp;
    }
    __syncthreads();
    const double total = tid < nslots ? s_out[tid] : 0.0;
    __syncthreads();  // the scratch may be reused by a following call
    return total;
}

}  // namespace gft
