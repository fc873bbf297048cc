// Host side of the register FFT engine (fft_reg.cuh, fft_reg.cu).
#pragma once

#include <vector>

#include "fft_reg.cuh"

struct iqm_ctx;

namespace iqm {

// Matrix bound: four sequences of a row pass stay within shared memory.
constexpr int REG_MAX_POINTS = 6144;

// A plan without tables: fills F (steps, sizes, kind) for length n; false when the engine has none.  Pure
// host code.
bool reg_plan(int n, RegFft &F, int &kind);

// The plan's estimated instructions a sequence takes.
long long reg_cost(const RegFft &F);

// The tables of a plan: one run of float2 holding twiddles, chirp and kernel, with their offsets.
struct RegTables {
    std::vector<float2> data;
    size_t chirp = 0, bhat = 0;
};
void reg_tables(const RegFft &F, RegTables &t);

// Threads of a CTA that transforms `count` sequences: the fewest (a multiple of 64, up to `most`) whose
// steps take the fewest rounds.  A round is a chain of loads, a DFT and stores, so idle lanes cost less
// than another round: inverse column pass of 270 points, 8 columns (144 and 120 lines a step), 64 pairs
// in chunks of two: 64 threads 755 us, 128 661, 160 621, 192 564, 256 623.
int reg_threads(const RegFft &F, int count, int most);

// The plan of length n with its device tables, made on first use and kept on the context (nullptr: none).
const RegFft *reg_fft_len(iqm_ctx *ctx, int n, int &kind);

}  // namespace iqm
