// FSIM forward transform on the register FFT engine: luma of a pair as Y_img + i Y_ref
// (src/gpu/fsim/fsim.cpp:270-368, sign -1, unscaled), rows then columns.  The column pass takes
// columns x and -x together, so that it can write each image's own spectrum:
// F(Y_img) = (Z(k) + conj Z(-k)) / 2, F(Y_ref) = (Z(k) - conj Z(-k)) / 2i.
#include "fsim_reg.cuh"

namespace iqm {

template <int KIND>
__global__ void __launch_bounds__(reg_most_threads(KIND), reg_min_ctas(KIND))
fsim_fwd_rows_reg(FsimGroup g, const __grid_constant__ RegFft F, int rows) {
    extern __shared__ __align__(16) float2 sm[];
    wait_for_previous();
    const int y0 = blockIdx.x * rows, pair = blockIdx.y;
    const float *Y1 = g.yiq + (size_t(pair * 2) * 3 + 2) * g.n + size_t(y0) * g.w2;
    const float *Y2 = Y1 + size_t(3) * g.n;
    float2 *Z = g.spec + size_t(pair) * g.n + size_t(y0) * g.w2;
    const int w2 = g.w2;
    const RowLayout lay{min(rows, g.h2 - y0), F.size, int(blockDim.x)};
    reg_fft<KIND>(
        F, lay, sm,
        [&](int seq, int i, int items) {
            const float *a = Y1 + (seq * w2 + i), *b = Y2 + (seq * w2 + i);
            const unsigned d = 4u * unsigned(items);
            return [=](int r) { return make_float2(__ldcg(run_at(b, d, r)), __ldcg(run_at(a, d, r))); };
        },
        [&](int seq, int i, int items) {
            float2 *z0 = Z + (seq * w2 + i);
            const unsigned d = 8u * unsigned(items);
            return [=](int r, unsigned, float2 v) { *run_at(z0, d, r) = make_float2(v.y, v.x); };
        });
}

template <int KIND>
__global__ void __launch_bounds__(reg_most_threads(KIND), reg_min_ctas(KIND))
fsim_fwd_cols_reg(FsimGroup g, const __grid_constant__ RegFft F, int lc) {
    extern __shared__ __align__(16) float2 sm[];
    wait_for_previous();
    const int half = 1 << (lc - 1);          // slots [0, half): columns x0 + c; the rest: columns -(x0 + c)
    const int x0 = blockIdx.x * half, pair = blockIdx.y;
    const int w2 = g.w2, h2 = g.h2;
    const int used = min(half, w2 / 2 + 1 - x0);
    const float2 *Z = g.spec + size_t(pair) * g.n;
    auto column = [&](int seq) {
        const int x = x0 + min(seq & (half - 1), used - 1);  // spare slots repeat the last column
        return seq < half ? x : (x ? w2 - x : 0);
    };
    const ColLayout<-1> lay{lc, 1 << lc, int(blockDim.x)};
    reg_fft<KIND>(
        F, lay, sm,
        [&](int seq, int i, int items) {
            const float2 *z0 = Z + (i * w2 + column(seq));
            const unsigned d = 8u * unsigned(items * w2);
            return [=](int r) {
                const float2 z = __ldcg(run_at(z0, d, r));
                return make_float2(z.y, z.x);
            };
        },
        [&](int, int, int) { return [](int, unsigned p, float2 v) { sts2(p, make_float2(v.y, v.x)); }; });
    __syncthreads();
    const RegStep &last = F.st[F.nsteps - 1];
    float2 *S1 = g.spec2 + size_t(pair) * g.spec_pair, *S2 = S1 + g.tiled;
    for (int w = threadIdx.x; w < (h2 << lc); w += blockDim.x) {
        const int seq = w & ((1 << lc) - 1), y = w >> lc;
        if ((seq & (half - 1)) >= used) continue;
        const float2 z = sm[lay.addr(seq, reg_out_addr(F, last, y))];
        const float2 m = sm[lay.addr(seq ^ half, reg_out_addr(F, last, y ? h2 - y : 0))];
        const int x = column(seq), at = (x >> g.lc) * g.tile + (y << g.lc) + (x & ((1 << g.lc) - 1));
        S1[at] = make_float2(0.5f * (z.x + m.x), 0.5f * (z.y - m.y));
        S2[at] = make_float2(0.5f * (z.y + m.y), 0.5f * (m.x - z.x));
    }
}

void launch_reg_fwd_rows(const FsimGroup &g, const FsimPlan &P, const RegShapes &s, cudaStream_t st) {
    with_kind(P.krow, [&](auto K) {
        auto fn = fsim_fwd_rows_reg<decltype(K)::value>;
        launch_transform(fn, dim3(ceil_div(P.h2, s.rows_f), g.G), s.t_fr, s.sm_fr, st, g, P.rrow, s.rows_f);
    });
}

void launch_reg_fwd_cols(const FsimGroup &g, const FsimPlan &P, const RegShapes &s, cudaStream_t st) {
    with_kind(P.kcol, [&](auto K) {
        auto fn = fsim_fwd_cols_reg<decltype(K)::value>;
        launch_transform(fn, dim3(ceil_div(P.w2 / 2 + 1, 1 << (s.lc_f - 1)), g.G), s.t_fc, s.sm_fc, st, g, P.rcol, s.lc_f);
    });
}

}  // namespace iqm
