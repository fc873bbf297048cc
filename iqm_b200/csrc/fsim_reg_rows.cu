// FSIM inverse transform, pass 2 (along x), on the register FFT engine, fused with the response sums of
// fsim_sum_filter_responses.glsl and fsim_pack_for_median.glsl: a CTA transforms the four scales of one
// orientation of `rows` rows, leaves the results in shared memory and sums them per pixel.  For a plan's
// constants (one row a CTA) it instead adds up, per row, sum_s Re_s^2 N and sum_{i<j} Re_i Re_j N
// (fsim_mult_filters.glsl:37-58) over p < ceil(N/2) and over all p.
#include "fsim_reg.cuh"

namespace iqm {

template <int KIND>
__global__ void __launch_bounds__(reg_most_threads(KIND), reg_min_ctas(KIND))
fsim_inv_rows_reg(FsimGroup g, const __grid_constant__ RegFft F, int rows, double *rowsums) {
    extern __shared__ __align__(16) float2 sm[];
    wait_for_previous();
    const int y0 = blockIdx.x * rows, o = blockIdx.y, plane = blockIdx.z;  // plane: chunk-local pair*2 + img
    const int w2 = g.w2;
    const int nr = min(rows, g.h2 - y0);
    const float2 *T = g.T + (size_t(plane) * 16 + o * 4) * g.n + size_t(y0) * w2;
    // sequence 4 row + scale
    const RowLayout lay{4 * nr, F.size, int(blockDim.x)};
    reg_fft<KIND>(
        F, lay, sm,
        [&](int seq, int i, int items) {
            const float2 *t0 = T + (size_t(seq & 3) * g.n + (seq >> 2) * w2 + i);
            const unsigned d = 8u * unsigned(items);
            return [=](int r) { return __ldcg(run_at(t0, d, r)); };
        },
        [&](int, int, int) { return [](int, unsigned p, float2 v) { sts2(p, v); }; });
    __syncthreads();
    const RegStep &last = F.st[F.nsteps - 1];
    if (!rowsums) {
        const size_t off = (size_t(g.pair0 * 2 + plane) * 4 + o) * g.n + size_t(y0) * w2;
        auto pixel = [&](int w, const float2 *p) {
            const float2 v[4] = {p[0], p[F.size], p[2 * F.size], p[3 * F.size]};
            float sA, en, e0;
            response_sums(v, sA, en, e0);
            __stcg(g.amp + off + w, sA);
            __stcg(g.energy + off + w, en);
            __stcg(g.eo0 + off + w, e0);
        };
        for (int rl = 0; rl < nr; rl++) {
            const float2 *row = sm + lay.addr(4 * rl, 0);
            if constexpr (KIND == REG_THREE) {
                for (int x = threadIdx.x; x < w2; x += blockDim.x) pixel(rl * w2 + x, row + reg_out_addr(F, last, x));
            } else {
                // output x = i + r items sits at i (hi or lo) + r stride: i and r advance with x
                const int step = last.d0 == 1 ? last.hi : last.lo;
                int r = div_by(threadIdx.x, F.inv_items_last), i = threadIdx.x - r * last.items;
                const int dr = div_by(blockDim.x, F.inv_items_last), di = blockDim.x - dr * last.items;
                for (int x = threadIdx.x; x < w2; x += blockDim.x) {
                    pixel(rl * w2 + x, row + i * step + r * last.stride);
                    r += dr;
                    i += di;
                    if (i >= last.items) {
                        i -= last.items;
                        r++;
                    }
                }
            }
        }
        return;
    }
    __shared__ double red[4][32];
    const long lim = (long(g.n) + 1) / 2;
    const float fn = float(g.n);
    double acc[4] = {0.0, 0.0, 0.0, 0.0};  // an2 (ref), aiaj (ref), an2 (full), aiaj (full)
    for (int x = threadIdx.x; x < w2; x += blockDim.x) {
        const float2 *p = sm + reg_out_addr(F, last, x);
        float re[4];
#pragma unroll
        for (int q = 0; q < 4; q++) re[q] = p[q * F.size].x;
        float q2 = 0.f, qx = 0.f;
#pragma unroll
        for (int q = 0; q < 4; q++) q2 += (re[q] * re[q]) * fn;
#pragma unroll
        for (int i = 0; i < 3; i++)
#pragma unroll
            for (int j = i + 1; j < 4; j++) qx += re[i] * re[j] * fn;
        if (long(y0) * w2 + x < lim) {
            acc[0] += q2;
            acc[1] += qx;
        }
        acc[2] += q2;
        acc[3] += qx;
    }
#pragma unroll
    for (int q = 0; q < 4; q++) {
        double v = acc[q];
        for (int d = 16; d > 0; d >>= 1) v += __shfl_down_sync(0xffffffffu, v, d);
        if ((threadIdx.x & 31) == 0) red[q][threadIdx.x >> 5] = v;
    }
    __syncthreads();
    if (threadIdx.x < 4) {
        double t = 0.0;
        for (int i = 0; i < int(blockDim.x) >> 5; i++) t += red[threadIdx.x][i];
        rowsums[(size_t(o) * g.h2 + y0) * 4 + threadIdx.x] = t;
    }
}

void launch_reg_inv_rows(const FsimGroup &g, const FsimPlan &P, const RegShapes &s, int planes, double *rowsums,
                         cudaStream_t st) {
    const int rows = rowsums ? 1 : s.rows_i;
    with_kind(P.krow, [&](auto K) {
        auto fn = fsim_inv_rows_reg<decltype(K)::value>;
        launch_transform(fn, dim3(ceil_div(P.h2, rows), 4, planes), s.t_ir, s.sm_ir, st, g, P.rrow, rows, rowsums);
    });
}

// Shared memory of the inverse column pass with 2^lc columns: matrices, spectrum tile, two filter tiles.
static size_t cols_smem(const FsimPlan &P, int lc, int tile) {
    return sizeof(float2) * (((size_t(P.rcol.size) << lc) + 1) & ~size_t(1)) + 16 * size_t(tile);
}

void reg_tiles(FsimPlan &P) {
    // eight columns (64-byte row segments of results) while two CTAs fit an SM, fewer for long columns
    for (P.lc = 3;; P.lc--) {
        P.tile = ((P.h2 << P.lc) + 3) & ~3;
        if (P.lc == 0 || cols_smem(P, P.lc, P.tile) <= 112 * 1024) break;
    }
    P.tiled = int(ceil_div(P.w2, 1 << P.lc)) * P.tile;
}

RegShapes reg_shapes(const FsimPlan &P, const FsimTune &tune) {
    RegShapes s{};
    const size_t f2 = sizeof(float2);
    const RegFft &R = P.rrow, &C = P.rcol;
    s.lc_f = std::max(1, P.lc);
    s.sm_ic = cols_smem(P, P.lc, P.tile);
    s.sm_fc = (size_t(C.size) << s.lc_f) * f2;
    s.t_ic = reg_threads(C, 1 << P.lc, reg_most_threads(P.kcol));
    s.t_fc = reg_threads(C, 1 << s.lc_f, reg_most_threads(P.kcol));
    // the inverse row pass holds four scales of a row
    s.rows_i = 8 * size_t(R.size) * f2 <= 64 * 1024 ? 2 : 1;
    if (tune.rows_per_cta == 1) s.rows_i = 1;
    s.sm_ir = 4 * size_t(s.rows_i) * R.size * f2;
    s.t_ir = reg_threads(R, 4 * s.rows_i, reg_most_threads(P.krow));
    s.rows_f = 8;
    while (s.rows_f > 1 && s.rows_f * size_t(R.size) * f2 > 64 * 1024) s.rows_f /= 2;
    s.sm_fr = s.rows_f * size_t(R.size) * f2;
    s.t_fr = reg_threads(R, s.rows_f, reg_most_threads(P.krow));
    return s;
}

}  // namespace iqm
