// SSIM / MSSIM on sm_100a: one fused kernel per batch of pairs.
//
// Reference path (cadik/IQM): three full-image Vulkan dispatches and a host pass --
//   luma pack        shaders/ssim/ssim_lumapack.glsl:19-35   (0.299 R + 0.581 G + 0.114 B, unorm)
//   Gaussian means   shaders/ssim/ssim_gaussinput.glsl:22-57 (11x11 window, truncated at the image
//                    border and renormalised by the in-image weight sum)
//   variances + map  shaders/ssim/ssim.glsl:25-79           (same window, two-pass form)
//   MSSIM            src/gpu/ssim/ssim.cpp:386-401           (x, y in [r, dim - r], host double sum)
//
// This kernel computes the same quantities in one pass over the RGBA8 inputs:
//   * the 2-D window is separable, w(dx,dy) = g(dx) g(dy), and so is its truncation: the in-image
//     weight sum of pixel (x,y) is wx(x) * wy(y);
//   * with u = a + b and v = a - b the five SSIM moments reduce to four (mean and second moment
//     of u and v): mu_a mu_b = (mu_u^2 - mu_v^2)/4, mu_a^2 + mu_b^2 = (mu_u^2 + mu_v^2)/2,
//     cov_ab = (var_u - var_v)/4, var_a + var_b = (var_u + var_v)/2;
//   * the second moments are taken about a per-tile constant (the u, v of the tile's centre
//     pixel), var = E[(x-c)^2] - E[x-c]^2, which keeps FP32 cancellation ~1e-7 on MSSIM;
//   * lumas stay whole numbers, 299 R + 581 G + 114 B, in units of 2^-18, so (u, v) and their distance to the
//     constant are exact in FP32 until the first tap multiplies them;
//   * each CTA owns a 128-column strip and streams down it four rows a step: the rows' (u, v) go to
//     shared memory, a warp a row filters them horizontally, four neighbouring columns a lane (a
//     staged value is loaded and squared once for the eleven outputs it serves), and a thread a column
//     runs the vertical taps as a transposed filter, whose running sums move up one register a row, so
//     that the row loop needs no unrolling over the window;
//   * (u, v) pairs are processed with packed FP32x2 instructions (__ffma2_rn and friends);
//   * MSSIM pools four rows of a column in FP32 and those sums in fixed point: neither the sum
//     nor any per-pixel value depends on how an image is cut into strips, which is chosen per launch
//     (strip_rows) from the number of images in it; the last CTA of a pair writes its mean.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <mutex>
#include <type_traits>

#include "iqm_internal.cuh"

namespace {

constexpr int TW = 128;             // output columns per CTA (one vertical strip)
constexpr int NT = TW;              // threads per CTA: a vertical column each
constexpr int RSTEP = 4;            // rows per step: a warp each in the horizontal pass
constexpr int UNITS = (TW + 16) / 2;  // staged columns x0-8 .. x0+TW+7 of a row, two to a 16-byte unit
constexpr int CHUNKS = (TW + 16) / 4; // 4-pixel loads of a row
constexpr int SHIFT_ROWS = 128;     // rows that share a shift constant; strips divide it
constexpr float LUMA_UNIT = 255000.0f / 262144.0f;  // a luma of 1 in the units used here: near 1, for the range of c1 and c2

struct Smem {
    float4 uv[RSTEP][UNITS];  // shifted (u, v) of two columns, at unit_at(flat index)
    float4 h[RSTEP][TW];      // horizontal sums (g u, g v, g u^2, g v^2), at column_at(column)
};

// Neighbouring lanes of the horizontal pass read every other unit and write every fourth column; these
// permutations spread them over the banks.
__device__ __forceinline__ int unit_at(int p) { return p ^ ((p >> 3) & 1); }
__device__ __forceinline__ int column_at(int c) { return c ^ ((c >> 3) & 3); }

struct SsimPairDev {
    const uint8_t *a;
    const uint8_t *b;
    float *map;        // nullable
    long long pitch;   // bytes between rows (both images)
    int w, h;
    int tiles_x;
    int tile_base;     // first global tile index of this pair
    int ntiles;
    int vec_ok;        // 16-byte loads allowed
};

struct SsimArgs {
    const SsimPairDev *pairs;
    int npairs;
    double *partials;    // one per tile
    unsigned *counters;  // one per pair, zero on entry
    double *scores;      // one per pair
    int strip;           // rows of a tile
    float2 g[8];         // 1-D Gaussian taps g(0..R), in both halves
    float c1, c2;        // in squared luma units
};

// shaders/ssim/ssim_lumapack.glsl:19-21 (G weight 0.581 as in the reference) times 255000: at most 253470.
__device__ __forceinline__ int luma_i(uint32_t px, int add) {
    return int(__dp2a_hi(114u, px, __dp2a_lo(299u | 581u << 16, px, unsigned(add))));
}
// (u, v) of a pixel pair as 48 + value * 2^-18 in floats, whose spacing there is 2^-18
__device__ __forceinline__ float2 uv_biased(uint32_t pa, uint32_t pb) {
    const int a = luma_i(pa, 0x42400000), b = luma_i(pb, 0);
    return make_float2(__int_as_float(a + b), __int_as_float(a - b));
}
constexpr float UV_BIAS = 48.0f;

__device__ __forceinline__ int find_pair(const SsimPairDev *pairs, int n, int tile) {
    int lo = 0, hi = n - 1;
    while (lo < hi) {
        int mid = (lo + hi + 1) >> 1;
        if (pairs[mid].tile_base <= tile) lo = mid; else hi = mid - 1;
    }
    return lo;
}

// Pooled values are sums of four rows' in units of 2^-37: a tile's 2^12 of them, below 8 each, are a whole
// number that FP64 holds.
constexpr double POOL_UNITS = 137438953472.0;

// Sum over the CTA, in a fixed order; valid in thread 0.  `red` holds NTH/32 values of 8 bytes.
template <int NTH, class T>
__device__ __forceinline__ T cta_sum(T v, double *red) {
    T *part = reinterpret_cast<T *>(red);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = v;
    __syncthreads();
    T s = 0;
#pragma unroll
    for (int i = 0; i < NTH / 32; i++) s += part[i];
    return s;
}

// Deterministic pooling: the CTA's partial goes to its tile slot; the last CTA of the pair to finish sums the
// pair's slots, in units (a pair's may pass 64 bits: the upper 40 and lower 24 bits of each tile's add up by
// themselves) so that neither the cut into tiles nor their order matters, and writes the mean (`count` pooled
// pixels).  Values that are no such numbers (too large, infinities and NaN) add up in FP64.
template <int NTH>
__device__ __forceinline__ void pool_tiles(double d, double *red, int *is_last, double *partials,
                                           unsigned *counters, double *scores, int pi, const SsimPairDev &P,
                                           int gt, double count) {
    const int tid = threadIdx.x;
    d = cta_sum<NTH>(d, red);
    if (tid == 0) {
        partials[gt] = d;
        __threadfence();
        const unsigned prev = atomicAdd(&counters[pi], 1u);
        *is_last = (prev == unsigned(P.ntiles - 1));
    }
    __syncthreads();
    if (!*is_last) return;
    __threadfence();
    long long hi = 0, lo = 0;
    double other = 0.0;
    for (int i = tid; i < P.ntiles; i += NTH) {
        const double v = __ldcg(&partials[P.tile_base + i]);
        if (fabs(v) <= 32768.0) {
            const long long u = __double2ll_rn(v * POOL_UNITS);
            hi += u >> 24;
            lo += u & 0xffffff;
        } else {
            other += v;
        }
    }
    hi = cta_sum<NTH>(hi, red);
    lo = cta_sum<NTH>(lo, red);
    other = cta_sum<NTH>(other, red);
    if (tid == 0) {
        scores[pi] = (double(hi) * (16777216.0 / POOL_UNITS) + double(lo) / POOL_UNITS + other) / count;
        counters[pi] = 0u;  // ready for the next launch
    }
}

// One thread's share of the staging: a 4-pixel chunk of both images in one row of every step.
struct Chunk {
    const uint8_t *a, *b;  // the chunk in the next step's row
    int y;                 // that row
    int nv;                // pixels of the chunk inside the image's columns
    int at;                // its first unit in Smem::uv
    uint4 ra, rb;

    __device__ __forceinline__ void init(const SsimPairDev &P, int xs, int yr, int c) {
        const int row = c / CHUNKS, q = c - row * CHUNKS, x = xs + 4 * q;
        y = yr + row;
        nv = x < 0 ? 0 : max(0, min(4, P.w - x));  // x is a multiple of 4: a chunk is all left of 0 or not at all
        a = P.a + (long long)y * P.pitch + 4LL * x;
        b = P.b + (long long)y * P.pitch + 4LL * x;
        at = row * UNITS + 2 * q;
    }
    // Reads the chunk (pixels outside the image are not read) and moves on to the next step's row.
    __device__ __forceinline__ void load(const SsimPairDev &P) {
        if (unsigned(y) < unsigned(P.h)) {
            if (P.vec_ok && nv == 4) {
                ra = __ldg(reinterpret_cast<const uint4 *>(a));
                rb = __ldg(reinterpret_cast<const uint4 *>(b));
            } else {
                const uint32_t *pa = reinterpret_cast<const uint32_t *>(a), *pb = reinterpret_cast<const uint32_t *>(b);
                if (nv > 0) ra.x = __ldg(pa), rb.x = __ldg(pb);
                if (nv > 1) ra.y = __ldg(pa + 1), rb.y = __ldg(pb + 1);
                if (nv > 2) ra.z = __ldg(pa + 2), rb.z = __ldg(pb + 2);
                if (nv > 3) ra.w = __ldg(pa + 3), rb.w = __ldg(pb + 3);
            }
        }
        a += RSTEP * P.pitch;
        b += RSTEP * P.pitch;
        y += RSTEP;
    }
    // Stores the shifted (u, v) of what was read; pixels outside the image become (0, 0), which removes
    // them from every window sum (the reference skips out-of-image taps).
    __device__ __forceinline__ void store(Smem &sm, int h, float2 shift) const {
        float2 v[4] = {__fadd2_rn(uv_biased(ra.x, rb.x), shift), __fadd2_rn(uv_biased(ra.y, rb.y), shift),
                       __fadd2_rn(uv_biased(ra.z, rb.z), shift), __fadd2_rn(uv_biased(ra.w, rb.w), shift)};
        const int n = unsigned(y - RSTEP) < unsigned(h) ? nv : 0;
        if (n < 4) {
#pragma unroll
            for (int k = 0; k < 4; k++)
                if (k >= n) v[k] = make_float2(0.f, 0.f);
        }
        float4 *uv = &sm.uv[0][0];
        uv[unit_at(at)] = make_float4(v[0].x, v[0].y, v[1].x, v[1].y);
        uv[unit_at(at + 1)] = make_float4(v[2].x, v[2].y, v[3].x, v[3].y);
    }
};

// Bound by the FMA pipe and instruction issue: of the instructions a pixel pair takes, 47 are the packed taps
// of both passes.  Four CTAs per SM at 125 registers, 16 1080p pairs: 214 us (236 us with a row's tests in
// every row instead of once a step; a Newton step on the quotient for identical images' sake took 217), against 397 us for the form before it (a column a thread, eleven loads and squares per pixel, the row loop
// unrolled over the window, a barrier a row; 297 instructions a pixel pair); five CTAs at 96 registers
// spill, 253 us.  The split-precision tensor-core form took 23.1 us a 1080p pair and the single-product
// one 15.6 us where this takes 13.3, so every form asked for computes here.
template <int R>
__global__ void __launch_bounds__(NT, 4) ssim_kernel(SsimArgs args) {
    constexpr int K = 2 * R + 1;
    __shared__ __align__(16) Smem sm;
    __shared__ double red[NT / 32];
    __shared__ int is_last;

    const int gt = blockIdx.x;
    const int pi = find_pair(args.pairs, args.npairs, gt);
    const SsimPairDev P = args.pairs[pi];
    const int local = gt - P.tile_base;
    const int x0 = (local % P.tiles_x) * TW;
    const int y0 = (local / P.tiles_x) * args.strip;
    const int W = P.w, H = P.h, xs = x0 - 8;
    const int y1 = min(y0 + args.strip, H);  // end of the strip's output rows
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

    // the strip's shift constants: u, v of the centre pixel of its block of SHIFT_ROWS rows
    float2 shift, c;
    {
        const int cx = min(x0 + TW / 2, W - 1), cy = min((y0 & ~(SHIFT_ROWS - 1)) + SHIFT_ROWS / 2, H - 1);
        shift = uv_biased(__ldg(reinterpret_cast<const uint32_t *>(P.a + (long long)cy * P.pitch) + cx),
                          __ldg(reinterpret_cast<const uint32_t *>(P.b + (long long)cy * P.pitch) + cx));
        c = make_float2(shift.x - UV_BIAS, shift.y - UV_BIAS);
        shift = make_float2(-shift.x, -shift.y);
    }
    auto tap = [&](int k) { return args.g[k < R ? R - k : k - R]; };  // g(k - R), symmetric
    const int x = x0 + tid;  // this thread's column of the vertical pass
    float rwx;               // 1 / in-image weight of the horizontal window
    {
        float s = 0.f;
#pragma unroll
        for (int k = 0; k < K; k++) s += (x + k - R >= 0 && x + k - R < W) ? tap(k).x : 0.f;
        rwx = 1.0f / s;
    }
    float gsum = args.g[0].x;
#pragma unroll
    for (int k = 1; k <= R; k++) gsum += 2.0f * args.g[k].x;
    const bool pool_x = x >= R && x <= W - R && x < W;

    float2 am[K - 1], as[K - 1];  // running vertical sums: element k waits for K - 1 - k more rows
#pragma unroll
    for (int k = 0; k < K - 1; k++) am[k] = as[k] = make_float2(0.f, 0.f);
    float acc = 0.f;     // pooled SSIM of up to four rows
    long long sum = 0;   // and of the strip, in POOL_UNITS
    double other = 0.0;  // sums that are no such numbers: k1 or k2 of 0 over flat areas
    auto pool = [&] {
        if (pool_x) {
            if (fabsf(acc) < 8.0f) sum += __float2ll_rn(acc * float(POOL_UNITS));
            else other += acc;
        }
        acc = 0.f;
    };

    const int yr = y0 - R;  // image row of the first staged row
    const int steps = (y1 - y0 + 2 * R + RSTEP - 1) / RSTEP;
    constexpr int EXTRA = RSTEP * CHUNKS - NT;  // chunks beyond one a thread
    Chunk first, second;
    first.init(P, xs, yr, tid);
    first.load(P);
    if (tid < EXTRA) {
        second.init(P, xs, yr, NT + tid);
        second.load(P);
    }
    first.store(sm, H, shift);
    if (tid < EXTRA) second.store(sm, H, shift);
    __syncthreads();

#pragma unroll 1
    for (int s = 0; s < steps; s++) {
        if (s + 1 < steps) {  // the next step's pixels arrive under this step's taps
            first.load(P);
            if (tid < EXTRA) second.load(P);
        }
        {
            // horizontal taps of row `warp`, columns 4 lane .. 4 lane + 3: staged columns 4 lane + 8 - R ..
            float2 hm[4], hs[4];
#pragma unroll
            for (int j = 0; j < 4; j++) hm[j] = hs[j] = make_float2(0.f, 0.f);
            constexpr int U0 = (8 - R) / 2, U1 = (8 + 3 + R) / 2;
#pragma unroll
            for (int u = U0; u <= U1; u++) {
                const float4 two = (&sm.uv[0][0])[unit_at(warp * UNITS + 2 * lane + u)];
#pragma unroll
                for (int e = 0; e < 2; e++) {
                    const int i = 2 * u + e - (8 - R);  // tap of column 0
                    if (i < 0 || i > K + 2) continue;
                    const float2 v = e ? make_float2(two.z, two.w) : make_float2(two.x, two.y);
                    const float2 q = __fmul2_rn(v, v);
#pragma unroll
                    for (int j = 0; j < 4; j++) {
                        if (i - j < 0 || i - j >= K) continue;
                        hm[j] = i == j ? __fmul2_rn(tap(0), v) : __ffma2_rn(tap(i - j), v, hm[j]);
                        hs[j] = i == j ? __fmul2_rn(tap(0), q) : __ffma2_rn(tap(i - j), q, hs[j]);
                    }
                }
            }
#pragma unroll
            for (int j = 0; j < 4; j++) sm.h[warp][column_at(4 * lane + j)] = make_float4(hm[j].x, hm[j].y, hs[j].x, hs[j].y);
        }
        __syncthreads();
        const int yo = yr + RSTEP * s - R;  // the output row that the step's first row completes
        // vertical taps; rows(plain): every row of the step completes an output row that is pooled, under a
        // whole window, and no map is wanted
        auto rows = [&](auto plain) {
#pragma unroll
            for (int i = 0; i < RSTEP; i++) {
                const float4 h = sm.h[i][column_at(tid)];
                const float2 h1 = make_float2(h.x, h.y), h2 = make_float2(h.z, h.w);
                const float2 mm = __ffma2_rn(tap(K - 1), h1, am[0]), ms = __ffma2_rn(tap(K - 1), h2, as[0]);
#pragma unroll
                for (int k = 0; k < K - 2; k++) {
                    am[k] = __ffma2_rn(tap(K - 2 - k), h1, am[k + 1]);
                    as[k] = __ffma2_rn(tap(K - 2 - k), h2, as[k + 1]);
                }
                am[K - 2] = __fmul2_rn(tap(0), h1);
                as[K - 2] = __fmul2_rn(tap(0), h2);
                const int y = yo + i;
                float wy = gsum;
                if constexpr (!decltype(plain)::value) {
                    if (y < y0 || y >= y1) continue;  // uniform, as all branches on y
                    if (y < R || y >= H - R) {
                        wy = 0.f;
#pragma unroll
                        for (int k = 0; k < K; k++) wy += (y + k - R >= 0 && y + k - R < H) ? tap(k).x : 0.f;
                    }
                }
                const float inv = rwx * iqm::rcp_approx(wy);
                const float2 sh = __fmul2_rn(mm, make_float2(inv, inv));  // shifted means
                const float varu = fmaf(ms.x, inv, -sh.x * sh.x), varv = fmaf(ms.y, inv, -sh.y * sh.y);
                const float2 mu = __fadd2_rn(sh, c), mu2 = __fmul2_rn(mu, mu);
                const float num = fmaf(0.5f, mu2.x - mu2.y, args.c1) * fmaf(0.5f, varu - varv, args.c2);
                const float den = fmaf(0.5f, mu2.x + mu2.y, args.c1) * fmaf(0.5f, varu + varv, args.c2);
                // den is about c1 c2 or more, but 0 is possible: k1 or k2 may be 0, and the variances round; inside
                // the reciprocal's range, 2^-126 to 2^126, as long as c1 c2 is.  A rounded product, so that no path
                // adds it unrounded to the pooled sum
                float ssim = __fmul_rn(num, iqm::rcp_approx(den));
                // equal numerator and denominator, as in identical images, make 1 without the reciprocal's error
                if (num == den) ssim = rintf(ssim);
                if constexpr (decltype(plain)::value) {
                    acc += ssim;
                } else {
                    if (P.map && x < W) P.map[(long long)y * W + x] = ssim;
                    if (y >= R && y <= H - R) acc += ssim;
                }
                if (((i - 2 * R) & 3) == 3) pool();  // y & 3 == 3: strips start at multiples of 4
            }
        };
        if (!P.map && yo >= max(y0, R) && yo + RSTEP <= min(y1, H - R)) rows(std::true_type{});
        else rows(std::false_type{});
        if (s + 1 < steps) {
            first.store(sm, H, shift);
            if (tid < EXTRA) second.store(sm, H, shift);
        }
        __syncthreads();
    }
    pool();
    pool_tiles<NT>(double(sum) * (1.0 / POOL_UNITS) + other, red, &is_last, args.partials, args.counters, args.scores, pi, P, gt,
                   double(W - 2 * R + 1) * double(H - 2 * R + 1));
}

}  // namespace

namespace {

template <int R>
void launch_ssim(const SsimArgs &a, int total_tiles, cudaStream_t s) {
    ssim_kernel<R><<<total_tiles, NT, 0, s>>>(a);
}

// Rows of a tile, the same for all pairs of a launch: the power of two that divides SHIFT_ROWS with the
// least estimated time, a tile's rows with its halo (and about a dozen rows' worth of set-up) times the
// rounds of two CTAs per SM that it takes.  The values of an image do not depend on the choice.  Strips
// of 8 / 16 / 32 / 64 / 128 rows: one 512x512 pair 15.3 / 15.3 / 18.1 / 25.2 / 37.5 us, one 1080p pair
// 42.0 / 31.8 / 29.8 / 29.7 / 38.0, four 131 / 92 / 74 / 66 / 71, 16 pairs 494 / 334 / 254 / 219 / 215 us.  Four
// CTAs run on an SM, but rounds of one, two or four choose within 2% of one another there, but for four 1080p
// pairs (71 / 71 / 66 us) and one of 720p (21.5 / 21.1 / 22.3 us).
int strip_rows(const iqm_pair *pairs, int n, int R) {
    int best = SHIFT_ROWS;
    double best_cost = 0.0;
    for (int s = SHIFT_ROWS; s >= 8; s /= 2) {
        double tiles = 0.0;
        for (int i = 0; i < n; i++) tiles += double(iqm::ceil_div(pairs[i].w, TW)) * iqm::ceil_div(pairs[i].h, s);
        const double cost = (s + 2 * R + 12) * std::max(1.0, tiles / (2 * 148));
        if (s == SHIFT_ROWS || cost < best_cost) {
            best = s;
            best_cost = cost;
        }
    }
    return best;
}

void check_params(const iqm_ssim_params &p) {
    int R = (p.kernel_size - 1) / 2;
    IQM_REQUIRE(R >= 1 && R <= 7, "kernel_size must give a radius (kernel_size-1)/2 in [1, 7]");
    IQM_REQUIRE(p.sigma > 0.f && std::isfinite(p.sigma), "sigma must be positive");
    IQM_REQUIRE(std::isfinite(p.k1) && std::isfinite(p.k2), "k1/k2 must be finite");
    IQM_REQUIRE(p.precision == IQM_FP32 || p.precision == IQM_MIXED || p.precision == IQM_MIXED_FAST,
                "unknown precision " + std::to_string(p.precision));
}

// Taps and constants of the kernel.
void set_constants(SsimArgs &a, const iqm_ssim_params &p, int R) {
    for (int k = 0; k < 8; k++) {
        const float g = k <= R ? float(std::exp(-double(k * k) / (2.0 * double(p.sigma) * p.sigma))) : 0.f;
        a.g[k] = make_float2(g, g);
    }
    a.c1 = p.k1 * p.k1 * (LUMA_UNIT * LUMA_UNIT);
    a.c2 = p.k2 * p.k2 * (LUMA_UNIT * LUMA_UNIT);
}

// Enqueue SSIM for device-resident pairs; `maps[i]` (device, nullable) receive the SSIM maps.
void ssim_enqueue(iqm_ctx *ctx, const std::vector<iqm_pair> &pairs, const iqm_ssim_params &p,
                  const std::vector<float *> &maps, double *d_scores) {
    const int n = int(pairs.size());
    const int R = (p.kernel_size - 1) / 2;
    const int strip = strip_rows(pairs.data(), n, R);
    std::vector<SsimPairDev> hd(n);
    int total = 0;
    for (int i = 0; i < n; i++) {
        const iqm_pair &q = pairs[i];
        SsimPairDev &d = hd[i];
        d.a = q.input;
        d.b = q.ref;
        d.map = maps.empty() ? nullptr : maps[i];
        d.pitch = (long long)q.row_bytes;
        d.w = q.w;
        d.h = q.h;
        d.tiles_x = int(iqm::ceil_div(q.w, TW));
        d.ntiles = d.tiles_x * int(iqm::ceil_div(q.h, strip));
        d.tile_base = total;
        d.vec_ok = ((reinterpret_cast<uintptr_t>(q.input) | reinterpret_cast<uintptr_t>(q.ref) |
                     uintptr_t(q.row_bytes)) & 15u) == 0;
        total += d.ntiles;
    }
    unsigned *counters = nullptr;
    auto *d_desc = static_cast<SsimPairDev *>(iqm::upload_with_counters(ctx, hd.data(), sizeof(SsimPairDev) * n, n, counters));
    auto *scr = static_cast<uint8_t *>(ctx->scratch.get(sizeof(double) * total, ctx->stream));
    SsimArgs a{};
    a.pairs = d_desc;
    a.npairs = n;
    a.partials = reinterpret_cast<double *>(scr);
    a.counters = counters;
    a.scores = d_scores;
    a.strip = strip;
    set_constants(a, p, R);
    switch (R) {
        case 1: launch_ssim<1>(a, total, ctx->stream); break;
        case 2: launch_ssim<2>(a, total, ctx->stream); break;
        case 3: launch_ssim<3>(a, total, ctx->stream); break;
        case 4: launch_ssim<4>(a, total, ctx->stream); break;
        case 5: launch_ssim<5>(a, total, ctx->stream); break;
        case 6: launch_ssim<6>(a, total, ctx->stream); break;
        default: launch_ssim<7>(a, total, ctx->stream); break;
    }
    iqm::check_launch(ctx, "ssim_kernel");
}

iqm_ssim_params resolve(const iqm_ssim_params *p) {
    iqm_ssim_params d;
    iqm_ssim_default_params(&d);
    return p ? *p : d;
}

}  // namespace

extern "C" __attribute__((visibility("default"))) void iqm_ssim_default_params(iqm_ssim_params *p) {
    if (!p) return;
    // src/gpu/ssim/ssim.h:31-34
    p->kernel_size = 11;
    p->k1 = 0.01f;
    p->k2 = 0.03f;
    p->sigma = 1.5f;
    p->precision = IQM_FP32;
}

void iqm::enqueue_ssim_dev(iqm_ctx *ctx, const iqm_pair *pairs, int n, const iqm_ssim_params *params,
                           double *d_scores) {
    const iqm_ssim_params p = resolve(params);
    check_params(p);
    const int R = (p.kernel_size - 1) / 2;
    iqm::check_pairs(pairs, n, R, R);
    iqm::check_dev_alignment(pairs, n);
    IQM_REQUIRE(d_scores != nullptr, "d_scores is NULL");
    ssim_enqueue(ctx, std::vector<iqm_pair>(pairs, pairs + n), p, {}, d_scores);
}

extern "C" __attribute__((visibility("default"))) int iqm_ssim_dev(iqm_ctx *ctx, const iqm_pair *pairs, int n, const iqm_ssim_params *params,
                            double *d_scores) {
    return iqm::guarded(ctx, [&] { iqm::enqueue_ssim_dev(ctx, pairs, n, params, d_scores); });
}

extern "C" __attribute__((visibility("default"))) int iqm_ssim_batch(iqm_ctx *ctx, const iqm_pair *pairs, int n, const iqm_ssim_params *params,
                              double *scores) {
    return iqm::guarded(ctx, [&] {
        const iqm_ssim_params p = resolve(params);
        check_params(p);
        const int R = (p.kernel_size - 1) / 2;
        iqm::check_pairs(pairs, n, R, R);
        IQM_REQUIRE(scores != nullptr, "scores is NULL");
        auto *d_scores = static_cast<double *>(ctx->scores.get(sizeof(double) * n, ctx->stream));
        iqm::upload_pipelined(ctx, pairs, n, [&](const iqm_pair *dev, int first, int count) {
            ssim_enqueue(ctx, std::vector<iqm_pair>(dev, dev + count), p, {}, d_scores + first);
        });
        IQM_CHECK_CUDA(cudaMemcpyAsync(scores, d_scores, sizeof(double) * n, cudaMemcpyDeviceToHost, ctx->stream));
        IQM_CHECK_CUDA(cudaStreamSynchronize(ctx->stream));
    });
}

extern "C" __attribute__((visibility("default"))) int iqm_ssim(iqm_ctx *ctx, const uint8_t *rgba_in, const uint8_t *rgba_ref, int w, int h,
                        size_t row_bytes, const iqm_ssim_params *params, float *map_out, double *mssim) {
    return iqm::guarded(ctx, [&] {
        const iqm_ssim_params p = resolve(params);
        check_params(p);
        IQM_REQUIRE(mssim != nullptr, "mssim is NULL");
        const int R = (p.kernel_size - 1) / 2;
        iqm_pair hp{rgba_in, rgba_ref, w, h, row_bytes};
        iqm::check_pairs(&hp, 1, R, R);
        auto dev = iqm::upload_pairs(ctx, &hp, 1);
        auto *d_score = static_cast<double *>(ctx->scores.get(sizeof(double), ctx->stream));
        std::vector<float *> maps;
        float *d_map = nullptr;
        if (map_out) {
            d_map = static_cast<float *>(ctx->maps.get(sizeof(float) * size_t(w) * h, ctx->stream));
            maps.push_back(d_map);
        }
        ssim_enqueue(ctx, dev, p, maps, d_score);
        IQM_CHECK_CUDA(cudaMemcpyAsync(mssim, d_score, sizeof(double), cudaMemcpyDeviceToHost, ctx->stream));
        if (map_out)
            IQM_CHECK_CUDA(cudaMemcpyAsync(map_out, d_map, sizeof(float) * size_t(w) * h,
                                           cudaMemcpyDeviceToHost, ctx->stream));
        IQM_CHECK_CUDA(cudaStreamSynchronize(ctx->stream));
    });
}

// ---------------------------------------------------------------------------------------------
// Allocation-free SSIM.  Some callers cannot let a library allocate device memory: a host
// application that reserves the whole GPU for its own allocator, or a plugin whose host accounts
// for every byte it hands out.  iqm_ssim_noalloc serves them: the caller passes device inputs and
// outputs, and the kernel's scratch (pair descriptor, completion counter, per-tile partial sums)
// lives in the fixed array below, which every GPU that loads this library holds until exit.
namespace {

struct NoallocScratch {
    SsimPairDev desc;                                 // the pair of the current call
    unsigned counter;                                 // CTAs finished; must be 0 at launch
    double partials[IQM_SSIM_NOALLOC_MAX_TILES];      // one per tile
};

static __device__ __align__(256) unsigned char g_ssim_noalloc_scratch[sizeof(NoallocScratch)];

// Host-side copies of the array's device address, one per device, filled on the first call made
// with that device current.  In host code the symbol itself is only a stand-in, not an address.
constexpr int NOALLOC_MAX_DEVICES = 64;
void *g_noalloc_addr[NOALLOC_MAX_DEVICES] = {};
std::mutex g_noalloc_mu;

// Writes the descriptor and clears the counter (the array keeps the previous call's contents).
__global__ void ssim_noalloc_setup_kernel(NoallocScratch *s, SsimPairDev d) {
    s->desc = d;
    s->counter = 0u;
}

// Launches ssim_kernel<R> and returns that launch's own status.  cudaLaunchKernel reports errors of
// this launch only, so an error left pending by the caller's earlier work is neither returned nor
// cleared here; a failed launch's own error is cleared before returning.
template <int R>
cudaError_t launch_ssim_checked(SsimArgs &a, int total_tiles, cudaStream_t st) {
    void *args[] = {&a};
    const cudaError_t e = cudaLaunchKernel((const void *)ssim_kernel<R>, dim3(total_tiles), dim3(NT), args, 0, st);
    if (e != cudaSuccess) cudaGetLastError();
    return e;
}

}  // namespace

extern "C" __attribute__((visibility("default"))) int iqm_ssim_noalloc(
    const uint8_t *d_in, const uint8_t *d_ref, int w, int h, size_t row_bytes, const iqm_ssim_params *params,
    float *d_map, double *d_mssim, void *cuda_stream) {
    if (!d_in || !d_ref || !d_mssim) return IQM_EINVAL;
    // pixels are read as 4-byte words, the score as a double and the map as floats: misaligned
    // pointers would fault on the GPU, so they are refused before any launch
    if (((reinterpret_cast<uintptr_t>(d_in) | reinterpret_cast<uintptr_t>(d_ref) | uintptr_t(row_bytes) |
          reinterpret_cast<uintptr_t>(d_map)) & 3u) != 0 || (reinterpret_cast<uintptr_t>(d_mssim) & 7u) != 0)
        return IQM_EINVAL;
    const iqm_ssim_params p = resolve(params);
    try {
        check_params(p);
    } catch (const iqm::Error &e) {
        return e.code;
    }
    if (p.precision != IQM_FP32) return IQM_EINVAL;  // the fixed scratch is sized for the FP32 tiles
    const int R = (p.kernel_size - 1) / 2;
    if (w < 2 * R || h < 2 * R || w > 65536 || h > 65536 || row_bytes < size_t(w) * 4) return IQM_EINVAL;
    const int tiles_x = int(iqm::ceil_div(w, TW));
    // the documented bound is in tiles of 120 to 127 rows (the 2R + 1 rows of a window divide a tile and
    // its halo); the kernel's own tiles of SHIFT_ROWS rows are never more
    const int bound_rows = (2 * R + 1) * int(iqm::ceil_div(120 + 2 * R, 2 * R + 1)) - 2 * R;
    if (long(tiles_x) * long(iqm::ceil_div(h, bound_rows)) > IQM_SSIM_NOALLOC_MAX_TILES) return IQM_EINVAL;
    // shorter strips for small images, as iqm_ssim takes them, while their sums fit the scratch
    const iqm_pair one{d_in, d_ref, w, h, row_bytes};
    int strip = strip_rows(&one, 1, R);
    while (strip < SHIFT_ROWS && long(tiles_x) * long(iqm::ceil_div(h, strip)) > IQM_SSIM_NOALLOC_MAX_TILES) strip *= 2;
    const long tiles = long(tiles_x) * long(iqm::ceil_div(h, strip));

    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= NOALLOC_MAX_DEVICES) return IQM_ECUDA;
    void *addr = nullptr;
    {
        std::lock_guard<std::mutex> lock(g_noalloc_mu);
        if (!g_noalloc_addr[dev]) {
            void *a = nullptr;
            if (cudaGetSymbolAddress(&a, g_ssim_noalloc_scratch) != cudaSuccess || !a) {
                cudaGetLastError();  // this lookup's own error
                return IQM_ECUDA;
            }
            g_noalloc_addr[dev] = a;
        }
        addr = g_noalloc_addr[dev];
    }
    auto *s = static_cast<NoallocScratch *>(addr);
    cudaStream_t st = static_cast<cudaStream_t>(cuda_stream);

    SsimPairDev d{};
    d.a = d_in;
    d.b = d_ref;
    d.map = d_map;
    d.pitch = (long long)row_bytes;
    d.w = w;
    d.h = h;
    d.tiles_x = tiles_x;
    d.tile_base = 0;
    d.ntiles = int(tiles);
    d.vec_ok = ((reinterpret_cast<uintptr_t>(d_in) | reinterpret_cast<uintptr_t>(d_ref) | uintptr_t(row_bytes)) &
                15u) == 0;
    {
        void *args[] = {&s, &d};
        const cudaError_t e =
            cudaLaunchKernel((const void *)ssim_noalloc_setup_kernel, dim3(1), dim3(1), args, 0, st);
        if (e != cudaSuccess) {
            cudaGetLastError();
            return IQM_ECUDA;  // the SSIM kernel is not launched without its descriptor
        }
    }

    SsimArgs a{};
    a.pairs = &s->desc;
    a.npairs = 1;
    a.partials = s->partials;
    a.counters = &s->counter;
    a.scores = d_mssim;
    a.strip = strip;
    set_constants(a, p, R);
    cudaError_t e;
    switch (R) {
        case 1: e = launch_ssim_checked<1>(a, int(tiles), st); break;
        case 2: e = launch_ssim_checked<2>(a, int(tiles), st); break;
        case 3: e = launch_ssim_checked<3>(a, int(tiles), st); break;
        case 4: e = launch_ssim_checked<4>(a, int(tiles), st); break;
        case 5: e = launch_ssim_checked<5>(a, int(tiles), st); break;
        case 6: e = launch_ssim_checked<6>(a, int(tiles), st); break;
        default: e = launch_ssim_checked<7>(a, int(tiles), st); break;
    }
    return e == cudaSuccess ? IQM_OK : IQM_ECUDA;
}
