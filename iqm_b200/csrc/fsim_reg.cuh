// FSIM's transform passes on the register FFT engine (fft_reg.cuh): launch interface.
#pragma once

#include <algorithm>

#include "fft_reg_plan.cuh"
#include "fsim_internal.cuh"

namespace iqm {

// Launch shapes of the four passes for one plane size.
struct RegShapes {
    int lc_f;              // log2 columns per CTA, forward column pass (inverse: FsimPlan::lc)
    int rows_f, rows_i;    // rows per CTA, forward and inverse row passes
    int t_fr, t_fc, t_ic, t_ir;  // threads per CTA
    size_t sm_fr, sm_fc, sm_ic, sm_ir;
};
RegShapes reg_shapes(const FsimPlan &P, const FsimTune &tune);
// Sets the plan's column tiles.
void reg_tiles(FsimPlan &P);

// Forward transform of G pairs: spec (packed, Y_img + i Y_ref) by rows, then columns into spec2, each
// image's own spectrum.
void launch_reg_fwd_rows(const FsimGroup &g, const FsimPlan &P, const RegShapes &s, cudaStream_t st);
void launch_reg_fwd_cols(const FsimGroup &g, const FsimPlan &P, const RegShapes &s, cudaStream_t st);
// The inverse passes of `planes` images from 2 g.pair0 on; g.T holds their 16 planes each.
void launch_reg_inv_cols(const FsimGroup &g, const FsimPlan &P, const RegShapes &s, int planes, cudaStream_t st);
// rowsums != nullptr: the transforms of the filters themselves, summed per row (plan constants).
void launch_reg_inv_rows(const FsimGroup &g, const FsimPlan &P, const RegShapes &s, int planes, double *rowsums,
                         cudaStream_t st);

// Raises a kernel's dynamic shared-memory limit on the current device to at least `bytes` (never lowers it);
// carveout: with the largest share of shared memory, for kernels that use no L1.
void set_smem(const void *fn, size_t bytes, bool carveout = true);

// Resident CTAs per SM of a kernel at a launch shape, memoised per device (raises the kernel's
// shared-memory limit first, as a launch would).
int resident_ctas(const void *fn, int threads, size_t smem, bool carveout = true);

// Launches a transform kernel with just the shared memory its resident CTAs use, so that the rest of the
// SM's array serves as L1 for the twiddles and for the spectrum that every scale reads again.
template <class... Params, class... Args>
inline void launch_transform(void (*fn)(Params...), dim3 grid, int threads, size_t smem, cudaStream_t st, const FsimGroup &g,
                             Args... args) {
    const int ctas = resident_ctas((const void *)fn, threads, smem, false);
    const size_t share = (ctas * (smem + 2048) * 100 + 228 * 1024 - 1) / (228 * 1024);
    launch_after(fn, grid, threads, smem, int(std::min<size_t>(100, share)), g.early, st, g, args...);
}

template <class F>
inline void with_kind(int kind, F &&f) {
    switch (kind) {
        case REG_DIRECT_24: f(std::integral_constant<int, REG_DIRECT_24>{}); break;
        case REG_DIRECT_32: f(std::integral_constant<int, REG_DIRECT_32>{}); break;
        case REG_BLUE_2: f(std::integral_constant<int, REG_BLUE_2>{}); break;
        case REG_BLUE_24: f(std::integral_constant<int, REG_BLUE_24>{}); break;
        default: f(std::integral_constant<int, REG_THREE>{}); break;
    }
}

// Threads a kernel of a kind may be launched with.
constexpr int reg_most_threads(int) { return 256; }
// CTAs of that many threads an SM has to hold: 80 registers a thread serve radices up to 24, 128 the rest.
constexpr int reg_min_ctas(int kind) { return kind == REG_DIRECT_32 || kind == REG_BLUE_2 ? 2 : 3; }

}  // namespace iqm
