// Declarations shared by FSIM's translation units: the plan of a plane size, the group of pairs that a
// launch works on, and the response sums.
#pragma once

#include "fft.cuh"
#include "fft_reg.cuh"
#include "iqm_internal.cuh"

namespace iqm {

struct FsimPlan {
    int w2 = 0, h2 = 0, n = 0;
    FftLen row{}, col{};       // shared-memory engine: planes with a side beyond the register engine
    bool reg = false;          // both sides run on the register engine
    RegFft rrow{}, rcol{};
    int krow = -1, kcol = -1;  // their RegKind
    // Spectrum and filter planes of the register engine are stored as tiles of 2^lc columns: element
    // (x, y) at (x >> lc) tile + (y << lc) + (x & (2^lc - 1)); `tiled` elements a plane.
    int lc = 0, tile = 0, tiled = 0;
    float *filters = nullptr;  // 16 planes of n (z = o*4 + s)
    double *consts = nullptr;  // device: em[4], an2[2][4], aiaj[2][4]
    double em[4], an2[2][4], aiaj[2][4];
    ~FsimPlan() {
        if (filters) cudaFree(filters);
        if (consts) cudaFree(consts);
    }
};

constexpr int FT = 256;  // threads per FFT / pointwise CTA

struct FsimPairDev {
    const uint8_t *a;
    const uint8_t *b;
    long long pitch;
    int w, h, F;
    int out;  // index of this pair in the caller's score array
};

struct FsimGroup {
    const FsimPairDev *pairs;
    int G;          // pairs in this launch
    int pair0;      // group index of the first pair of this launch (inverse-pass chunks)
    int w2, h2, n;
    float *yiq;     // G x 2 x 3 x n   (I, Q, Y)
    float2 *spec;   // G x n: per pair the spectrum of Y_img + i Y_ref
    float2 *spec2;  // per pair, spec_pair apart, 2 x tiled: each image's own spectrum (register engine)
    size_t spec_pair;
    int lc, tile, tiled;  // FsimPlan's
    float2 *T;      // chunk x 2 x 16 x n  (after the column pass of the inverse transform)
    float *amp;     // G x 8 x n       (img*4 + o)
    float *energy;  // G x 8 x n
    float *eo0;     // G x 8 x n       |EO(s=0, o)|^2
    float *thr;     // G x 8
    double *partials;  // G x tiles x 3
    unsigned *counters;
    int tiles;
    bool early;     // launch_after's
    double *scores;    // 2 per pair: fsim, fsimc
    const float *filters;  // 16 planes, tiled (register engine), else column-major x * h2 + y
    const double *consts;
    int energy_mode;
};

// A kernel of FSIM's chain may be launched while the one before it in its stream still drains (launch_after);
// it calls this before it touches memory and goes on when that one's writes are visible.  What another kernel
// of the chain writes is not read with __ldg, whose memory must not change while the kernel runs: this one runs
// from its launch on, when that memory is still being written.  Plan tables may be.
__device__ __forceinline__ void wait_for_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Launches a kernel that calls wait_for_previous(): its CTAs are set up during the tail of the stream's
// previous kernel, which saves a launch latency per kernel of a chain of short ones.
// carveout > 0: the share of the SM's array kept as shared memory, in percent.  early = false: after the
// previous kernel's end as usual.  One 512x384 pair 73 us, with early launches 58.  Where chunks of pairs alternate
// between two streams, whose kernels fill much of each other's tails, they are not used yet, though they gain
// there as well: 32 1080p pairs 999.6 us, with early launches 985.6.
template <class... Params, class... Args>
inline void launch_after(void (*fn)(Params...), dim3 grid, int threads, size_t smem, int carveout, bool early, cudaStream_t st,
                         Args... args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[2]{};
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = early ? 1 : 0;
    attr[1].id = cudaLaunchAttributePreferredSharedMemoryCarveout;
    attr[1].val.sharedMemCarveout = unsigned(carveout);
    cfg.attrs = attr;
    cfg.numAttrs = carveout > 0 ? 2 : 1;
    IQM_CHECK_CUDA(cudaLaunchKernelEx(&cfg, fn, Params(args)...));
}

// Per-pixel response sums of one orientation from its 4 normalised scales, as
// shaders/fsim/fsim_sum_filter_responses.glsl:43-80 and fsim_pack_for_median.glsl:39-43; square
// roots and the reciprocal from the SFU approximations.
__device__ __forceinline__ void response_sums(const float2 v[4], float &sA, float &en, float &e0) {
    float sE = 0.f, sO = 0.f, e[4];
    sA = 0.f;
#pragma unroll
    for (int s = 0; s < 4; s++) {
        e[s] = v[s].x * v[s].x + v[s].y * v[s].y;
        sA += sqrt_approx(e[s]);
        sE += v[s].x;
        sO += v[s].y;
    }
    const float rxe = rcp_approx(sqrt_approx(sE * sE + sO * sO) + 0.0001f);
    const float mE = sE * rxe, mO = sO * rxe;
    en = 0.f;
#pragma unroll
    for (int s = 0; s < 4; s++) en += v[s].x * mE + v[s].y * mO - fabsf(v[s].x * mO - v[s].y * mE);
    e0 = e[0];
}
}  // namespace iqm
