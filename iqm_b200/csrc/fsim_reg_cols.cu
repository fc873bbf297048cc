// FSIM inverse transform, pass 1 (along y), on the register FFT engine: an image's spectrum times
// H[o*4 + s] (fsim_filter_combinations.glsl:53-56), sign +1.
//
// A CTA takes a tile of 2^lc columns of one image and the four scales of one orientation.  Spectrum and
// filters are stored tile by tile (FsimPlan::tile), so a tile is one contiguous run: the spectrum's tile
// is copied to shared memory once, with asynchronous 16-byte copies, and each filter's tile while the
// scale before it is transformed.  Nothing but the results then passes through the L1 (as plain loads
// of 32- and 64-byte row segments, spectrum and filters kept it 76% busy and the lines did not survive
// from one scale to the next: 412 us a step of 64 1080p-sized images in launches of 16).
#include "fsim_reg.cuh"

namespace iqm {

__device__ __forceinline__ void copy16(unsigned dst, const void *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
// Starts copying `bytes` (a multiple of 16, both ends 16-byte aligned) to shared memory.
__device__ __forceinline__ void copy_run(unsigned dst, const void *src, int bytes) {
    for (int b = 16 * threadIdx.x; b < bytes; b += 16 * blockDim.x) copy16(dst + b, static_cast<const char *>(src) + b);
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void copy_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

template <int KIND, int LC>
__global__ void __launch_bounds__(reg_most_threads(KIND), reg_min_ctas(KIND))
fsim_inv_cols_reg(FsimGroup g, const __grid_constant__ RegFft F, int lc_) {
    const int lc = LC >= 0 ? LC : lc_;
    extern __shared__ __align__(16) float2 sm[];  // matrices, spectrum tile, two filter tiles
    const int o = blockIdx.y, plane = blockIdx.z;  // plane: chunk-local pair*2 + img
    const int x0 = blockIdx.x << lc, w2 = g.w2;
    const float2 *S = g.spec2 + size_t(g.pair0 + (plane >> 1)) * g.spec_pair + size_t(plane & 1) * g.tiled + size_t(blockIdx.x) * g.tile;
    const float *H = g.filters + size_t(o * 4) * g.tiled + size_t(blockIdx.x) * g.tile;
    const unsigned s_tile = smem_addr(sm) + 8u * (((F.size << lc) + 1) & ~1), h_tile = s_tile + 8u * g.tile;
    copy_run(h_tile, H, 4 * g.tile);  // the plan's, not the previous kernel's
    wait_for_previous();
    copy_run(s_tile, S, 8 * g.tile);
    copy_commit();
    const ColLayout<LC> lay{lc, min(1 << lc, w2 - x0), int(blockDim.x)};
    for (int s = 0; s < 4; s++) {
        const unsigned h_now = h_tile + (s & 1) * 4u * g.tile;
        if (s < 3) {  // into the tile that scale s - 1 read
            copy_run(h_tile + ((s + 1) & 1) * 4u * g.tile, H + size_t(s + 1) * g.tiled, 4 * g.tile);
            copy_commit();
            copy_wait<1>();
        } else {
            copy_wait<0>();
        }
        __syncthreads();  // the tiles are there, and the previous scale's lines are read
        float2 *T = g.T + (size_t(plane) * 16 + o * 4 + s) * g.n + x0;
        reg_fft<KIND>(
            F, lay, sm,
            [&](int seq, int i, int items) {
                const unsigned at = (i << lc) + seq, d = items << lc;
                return [=](int r) {
                    const float2 v = lds2(s_tile + 8u * at + r * (8u * d));
                    const float h = lds1(h_now + 4u * at + r * (4u * d));
                    return make_float2(h * v.x, h * v.y);
                };
            },
            [&](int seq, int i, int items) {
                float2 *t0 = T + (i * w2 + seq);
                const unsigned d = 8u * unsigned(items * w2);
                return [=](int r, unsigned, float2 v) { __stcg(run_at(t0, d, r), v); };
            });
    }
}

void launch_reg_inv_cols(const FsimGroup &g, const FsimPlan &P, const RegShapes &s, int planes, cudaStream_t st) {
    with_kind(P.kcol, [&](auto K) {
        auto fn = P.lc == 3 ? fsim_inv_cols_reg<decltype(K)::value, 3> : fsim_inv_cols_reg<decltype(K)::value, -1>;
        launch_transform(fn, dim3(ceil_div(P.w2, 1 << P.lc), 4, planes), s.t_ic, s.sm_ic, st, g, P.rcol, P.lc);
    });
}

}  // namespace iqm
