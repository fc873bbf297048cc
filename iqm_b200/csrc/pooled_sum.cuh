// Sums of FP32 values that do not depend on how they are split over threads and CTAs: fixed point of 2^-47,
// which holds every value of 2^-23 and above to its last bit and is 2^-48 off below that, in 64-bit integers.
#pragma once

#include <cuda_runtime.h>

namespace iqm {

struct PooledSum {
    long long units = 0;  // of 2^-47; up to 2^14 values of size 4 fit
    double other = 0.0;   // values that are no such numbers (larger ones, infinities and NaN)
    __device__ __forceinline__ void add(float v) {
        if (fabsf(v) < 4.0f) units += __float2ll_rn(v * 140737488355328.0f);
        else other += v;
    }
};

// Pools the CTA's sum (of at most 2^14 values) into tile slot gt of pair pi; the last CTA of the pair's
// `ntiles` (slots from tile_base on) writes the mean of `count` values and resets the pair's counter.
// Returns after a barrier only if the CTA is not the last one.
template <int NTH>
__device__ __forceinline__ void pool_tiles(PooledSum s, PooledSum *partials, unsigned *counters, double *scores, int pi, int gt,
                                           int tile_base, int ntiles, double count) {
    __shared__ PooledSum red[NTH / 32];
    __shared__ int is_last;
    const int tid = threadIdx.x;
    auto cta_sum = [&](long long &a, double &b) {  // over the CTA, in a fixed order; valid in thread 0
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            a += __shfl_down_sync(0xffffffffu, a, o);
            b += __shfl_down_sync(0xffffffffu, b, o);
        }
        if ((tid & 31) == 0) {
            red[tid >> 5].units = a;
            red[tid >> 5].other = b;
        }
        __syncthreads();
        if (tid == 0) {
            a = 0;
            b = 0.0;
            for (int i = 0; i < NTH / 32; i++) {
                a += red[i].units;
                b += red[i].other;
            }
        }
    };
    cta_sum(s.units, s.other);
    if (tid == 0) {
        partials[gt] = s;
        __threadfence();
        const unsigned prev = atomicAdd(&counters[pi], 1u);
        is_last = prev == unsigned(ntiles - 1);
    }
    __syncthreads();
    if (!is_last) return;
    __threadfence();
    // a pair's units may pass 64 bits: the upper 40 and lower 24 bits of each tile's add up by themselves
    long long hi = 0, lo = 0;
    double other = 0.0, none = 0.0;
    for (int i = tid; i < ntiles; i += NTH) {
        const long long u = __ldcg(&partials[tile_base + i].units);
        hi += u >> 24;
        lo += u & 0xffffff;
        other += __ldcg(&partials[tile_base + i].other);
    }
    cta_sum(hi, other);
    __syncthreads();
    cta_sum(lo, none);
    if (tid == 0) {
        scores[pi] = (double(hi) * (1.0 / 8388608.0) + double(lo) * (1.0 / 140737488355328.0) + other) / count;
        counters[pi] = 0u;  // ready for the next launch
    }
}

}  // namespace iqm
