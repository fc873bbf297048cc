// M-SVD on sm_100a.
//
// Reference path (cadik/IQM, src/gpu/svd/svd.cpp:39-164): on the host, OpenCV grey conversion
// (cv::cvtColor RGB2GRAY, uint8) and cv::SVD(NO_UV) of every 8x8 block of both images, for blocks
// with x+8 < W and y+8 < H only; on the GPU, the per-block distance D = sqrt(sum_k (s_k - r_k)^2)
// (shaders/svd/svd.glsl:24-54); on the host again a sort, the median D[n/2] and
// msvd = sum |D - median| / n with n = (W/8)*(H/8) (skipped slots count as D = 0).
//
// Here everything runs on the device in two kernels:
//   msvd_block_kernel  two lanes per block slot (one per image): 8 rows x 8 RGBA8 pixels straight
//                      into registers (two 16-byte loads per row, coalesced across a warp of
//                      horizontally adjacent blocks), OpenCV's 15-bit fixed-point grey, singular
//                      values in registers by bidiagonalisation (two rows per packed FP32x2
//                      instruction) and differential qd sweeps, D in FP32 as the shader does;
//   msvd_pool_kernel   one CTA per pair: exact median by radix select (select.cuh), then the mean
//                      absolute deviation summed in FP64, and the optional D/max(D) map.
#include <cfloat>
#include <cmath>

#include "iqm_internal.cuh"
#include "packed_f32x2.cuh"
#include "select.cuh"

namespace {

constexpr int BLOCK_THREADS = 128;
constexpr int POOL_THREADS = 1024;

struct MsvdPairDev {
    const uint8_t *a;
    const uint8_t *b;
    float *map;          // nullable, bw*bh
    long long pitch;
    int w, h;
    int bw, bh;          // W/8, H/8 block slots
    int vx, vy;          // computed blocks per row / column (x+8 < W, y+8 < H)
    int slot_base;       // first global slot of this pair
    int vec_ok;
};

struct MsvdArgs {
    const MsvdPairDev *pairs;
    int npairs;
    int total_slots;
    float *dist;         // total_slots
    double *scores;      // npairs
};

// cv::cvtColor(COLOR_RGB2GRAY) on 8-bit data: (R*9798 + G*19235 + B*3735 + 2^14) >> 15, in [0, 255], as
// 2^23 + value: the weighted sum is two 16-by-8-bit dot products (the alpha byte weighs 0), and the
// funnel shift that drops its 15 low bits brings the exponent of 2^23 in from above.
__device__ __forceinline__ float gray_plus_2p23(uint32_t px) {
    unsigned s = __dp2a_lo(9798u | 19235u << 16, px, 16384u);
    s = __dp2a_hi(3735u, px, s);
    return __uint_as_float(__funnelshift_r(s, 0x4B000000u >> 17, 15));
}

__device__ __forceinline__ int find_pair(const MsvdPairDev *p, int n, int slot) {
    int lo = 0, hi = n - 1;
    while (lo < hi) {
        int mid = (lo + hi + 1) >> 1;
        if (p[mid].slot_base <= slot) lo = mid; else hi = mid - 1;
    }
    return lo;
}

// Loads one 8x8 grey block, column-major in registers as row pairs: c[col][k] = (row 2k, row 2k + 1).
__device__ __forceinline__ void load_block(const uint8_t *img, long long pitch, int x, int y, bool vec,
                                           float2 c[8][4]) {
#pragma unroll
    for (int r = 0; r < 8; r++) {
        const uint8_t *row = img + (long long)(y + r) * pitch + 4LL * x;
        uint32_t px[8];
        if (vec) {
            const uint4 lo = __ldg(reinterpret_cast<const uint4 *>(row));
            const uint4 hi = __ldg(reinterpret_cast<const uint4 *>(row) + 1);
            px[0] = lo.x; px[1] = lo.y; px[2] = lo.z; px[3] = lo.w;
            px[4] = hi.x; px[5] = hi.y; px[6] = hi.z; px[7] = hi.w;
        } else {
#pragma unroll
            for (int q = 0; q < 8; q++) px[q] = __ldg(reinterpret_cast<const uint32_t *>(row) + q);
        }
#pragma unroll
        for (int q = 0; q < 8; q++) {
            if (r & 1) c[q][r >> 1].y = gray_plus_2p23(px[q]);
            else c[q][r >> 1].x = gray_plus_2p23(px[q]);
        }
    }
#pragma unroll
    for (int q = 0; q < 8; q++)
#pragma unroll
        for (int k = 0; k < 4; k++) c[q][k] = iqm::add2(c[q][k], iqm::dup2(-8388608.0f));
}

// A Householder reflection I - beta v v' that takes a vector of squared norm nn and first element x0 to
// (alpha, 0, ...): v is the vector with x0 - alpha in place of x0.  A vector of zeros is left as it is
// (beta 0), which also covers vectors of rounding noise too small for the squares of FP32.
__device__ __forceinline__ void reflection(float nn, float x0, float &alpha, float &beta) {
    const bool live = nn > 1e-30f;
    const float norm = iqm::sqrt_newton(fmaxf(nn, 1e-30f));
    alpha = live ? -copysignf(norm, x0) : 0.0f;
    beta = live ? iqm::rcp_newton(fmaf(fabsf(x0), norm, nn)) : 0.0f;
}

// Step K of the bidiagonalisation: column K is reflected to its diagonal element d, then row K right of
// it to e (the next two columns' element).  Rows go two to a register pair; rows above K in a pair that
// straddles it are dead and may take any value.
template <int K>
__device__ __forceinline__ void bidiagonal_step(float2 (&c)[8][4], float (&d)[8], float (&e)[7]) {
    if constexpr (K < 7) {
        constexpr int P0 = K >> 1;  // first pair with rows >= K
        float2 v[4];
#pragma unroll
        for (int p = P0; p < 4; p++) v[p] = c[K][p];
        if (K & 1) v[P0].x = 0.f;
        float2 n2 = iqm::mul2(v[P0], v[P0]);
#pragma unroll
        for (int p = P0 + 1; p < 4; p++) n2 = iqm::fma2(v[p], v[p], n2);
        float beta;
        const float x0 = (K & 1) ? v[P0].y : v[P0].x;
        reflection(n2.x + n2.y, x0, d[K], beta);
        if (K & 1) v[P0].y = x0 - d[K];
        else v[P0].x = x0 - d[K];
#pragma unroll
        for (int j = K + 1; j < 8; j++) {
            float2 s2 = iqm::mul2(v[P0], c[j][P0]);
#pragma unroll
            for (int p = P0 + 1; p < 4; p++) s2 = iqm::fma2(v[p], c[j][p], s2);
            const float2 s = iqm::dup2(-beta * (s2.x + s2.y));
#pragma unroll
            for (int p = P0; p < 4; p++) c[j][p] = iqm::fma2(s, v[p], c[j][p]);
        }
    } else {
        d[7] = c[7][3].y;
    }
    if constexpr (K < 6) {
        constexpr int R = K >> 1, P0 = (K + 1) >> 1;  // row K's pair, first pair with rows > K
        float v[8];
        float nn = 0.f;
#pragma unroll
        for (int j = K + 1; j < 8; j++) {
            v[j] = (K & 1) ? c[j][R].y : c[j][R].x;
            nn = fmaf(v[j], v[j], nn);
        }
        float beta;
        reflection(nn, v[K + 1], e[K], beta);
        v[K + 1] -= e[K];
        float2 s[4];
#pragma unroll
        for (int j = K + 1; j < 8; j++)
#pragma unroll
            for (int p = P0; p < 4; p++)
                s[p] = j == K + 1 ? iqm::mul2(iqm::dup2(v[j]), c[j][p]) : iqm::fma2(iqm::dup2(v[j]), c[j][p], s[p]);
#pragma unroll
        for (int p = P0; p < 4; p++) s[p] = iqm::mul2(s[p], iqm::dup2(-beta));
#pragma unroll
        for (int j = K + 1; j < 8; j++)
#pragma unroll
            for (int p = P0; p < 4; p++) c[j][p] = iqm::fma2(iqm::dup2(v[j]), s[p], c[j][p]);
    } else if constexpr (K == 6) {
        e[6] = c[7][3].x;
    }
}

// State of the quotient-difference iteration on the squares q of the diagonal and e of the superdiagonal.
struct QdState {
    float q[8], e[7];
    float sigma;     // shifts applied so far: an eigenvalue is sigma + its q
    float s1, s2;    // sums of 1 / x and 1 / x^2 over the eigenvalues of all rows but the last swept one
    bool converged;  // no value ran out of sweeps
};

// No e goes below this.  An exact 0 would split the matrix, and a pivot of 0 above it (a block whose first
// row and column are black) would make the step across it 0 / 0 and lose the value behind it; with it a
// pivot of 0 passes its neighbour's q on through e and moves down a row, and sweeps of split matrices bring
// the smallest value to the end like any other.  As a superdiagonal element it is 1e-10, which moves no
// singular value by more than that.
constexpr float kSmallestE = 1e-20f;
// The last row splits off below this: as a superdiagonal element 1e-4, which is also the most that leaving it
// out can move a singular value (and moves it by its square over twice the gap to the next one).  A bound
// that grows with the value, e <= 1e-5 x, let close values move by up to 1e-2; asking for the gap as well
// cost more than the sweep that the last digits take (209 us for 16 1080p pairs; with gaps 223 and above).
constexpr float kNegligibleE = 1e-8f;
constexpr int kMostSweeps = 24;  // of one value; about three in 10^5 noisy diagonal blocks need more

// Laguerre's lower bound of the smallest of m positive numbers whose reciprocals and their squares sum to
// s1 and s2, a little less; 0 where the sums are not usable.
__device__ __forceinline__ float laguerre_shift(float m, float s1, float s2) {
    const float root = iqm::sqrt_approx(fmaxf((m - 1.0f) * fmaf(m, s2, -s1 * s1), 0.0f));
    const float t = 0.9999f * m * iqm::rcp_approx(s1 + root);
    return t > 1e-6f ? t : 0.0f;  // below 1e-6 (a singular value of 1e-3) the plain iteration converges at once
}

// Finds the smallest eigenvalue of the leading M rows and leaves it in q[M - 1] + sigma: shifted
// differential qd sweeps until the last row splits off.
// Every sweep also carries the first two derivatives of its pivots by the shift, which give the sums over
// 1 / x and 1 / x^2 of the swept matrix's eigenvalues and with them the next shift; the sums without the
// last pivot are those of the matrix that is left when the last row splits off.
template <int M>
__device__ __forceinline__ void qd_smallest(QdState &z) {
    float tau = M == 8 ? 0.0f : laguerre_shift(float(M), z.s1, z.s2);
#pragma unroll 1
    for (int it = 0; z.e[M - 2] > kNegligibleE; it++) {
        if (it == kMostSweeps) {
            z.converged = false;
            break;
        }
        float Q[M], E[M - 1];
        float dd = z.q[0] - tau, low = dd, d1 = -1.0f, d2 = 0.0f, s1 = 0.0f, s2 = 0.0f;
#pragma unroll
        for (int i = 0; i < M - 1; i++) {
            Q[i] = dd + z.e[i];  // at least kSmallestE unless the shift is rejected below
            const float r = iqm::rcp_approx(Q[i]);
            const float t = z.q[i + 1] * r;
            E[i] = fmaxf(z.e[i] * t, kSmallestE);
            const float a = d1 * r, w = E[i] * r;
            s1 -= a;
            s2 = fmaf(-d2, r, fmaf(a, a, s2));
            d2 = w * fmaf(-2.0f * a, d1, d2);
            d1 = fmaf(w, d1, -1.0f);
            dd = fmaf(dd, t, -tau);
            low = fminf(low, dd);
        }
        Q[M - 1] = dd;
        if (low >= 0.0f) {
#pragma unroll
            for (int i = 0; i < M; i++) z.q[i] = Q[i];
#pragma unroll
            for (int i = 0; i < M - 1; i++) z.e[i] = E[i];
            z.sigma += tau;
            z.s1 = s1;
            z.s2 = s2;
            const float r = iqm::rcp_approx(fmaxf(dd, kSmallestE)), a = d1 * r;
            tau = laguerre_shift(float(M), s1 - a, fmaf(-d2, r, fmaf(a, a, s2)));
        } else {
            tau = 0.0f;  // the shift passed the smallest eigenvalue: sweep again without one
        }
    }
    z.q[M - 1] += z.sigma;
}

// Singular values of the 8x8 matrix whose columns are c[0..7], in no order; c is destroyed.  False where
// the iteration ran out of sweeps.
// Householder reflections to bidiagonal form, then the singular values of that by shifted differential
// qd sweeps (K. V. Fernando and B. N. Parlett, "Accurate singular values and differential qd algorithms",
// 1994), smallest first, with Laguerre's shifts.
__device__ __forceinline__ bool svd8_qd(float2 (&c)[8][4], float (&s)[8]) {
    QdState z;
    {
        float d[8], e[7];
        bidiagonal_step<0>(c, d, e);
        bidiagonal_step<1>(c, d, e);
        bidiagonal_step<2>(c, d, e);
        bidiagonal_step<3>(c, d, e);
        bidiagonal_step<4>(c, d, e);
        bidiagonal_step<5>(c, d, e);
        bidiagonal_step<6>(c, d, e);
        bidiagonal_step<7>(c, d, e);
#pragma unroll
        for (int i = 0; i < 8; i++) z.q[i] = d[i] * d[i];
#pragma unroll
        for (int i = 0; i < 7; i++) z.e[i] = fmaxf(e[i] * e[i], kSmallestE);
    }
    z.sigma = z.s1 = z.s2 = 0.0f;
    z.converged = true;
    qd_smallest<8>(z);
    qd_smallest<7>(z);
    qd_smallest<6>(z);
    qd_smallest<5>(z);
    qd_smallest<4>(z);
    qd_smallest<3>(z);
    qd_smallest<2>(z);
    z.q[0] += z.sigma;
#pragma unroll
    for (int i = 0; i < 8; i++) s[i] = z.q[i] > 1e-30f ? iqm::sqrt_newton(z.q[i]) : 0.0f;
    return z.converged;
}

// <ci, cj> over the 8 rows
__device__ __forceinline__ float dot8(const float2 (&ci)[4], const float2 (&cj)[4]) {
    float2 q = iqm::mul2(ci[0], cj[0]);
#pragma unroll
    for (int k = 1; k < 4; k++) q = iqm::fma2(ci[k], cj[k], q);
    return q.x + q.y;
}

// The same by one-sided Jacobi rotations, which need no shifts and converge on every block: for those that
// ran out of sweeps.  Each pair of columns is rotated so that they become orthogonal, until no inner product
// is above FP32's rounding of the two norms; the final norms are summed in FP64.
__device__ __forceinline__ void svd8_jacobi(float2 (&c)[8][4], float (&s)[8]) {
    const float eps2 = 16.0f * FLT_EPSILON * FLT_EPSILON;
#pragma unroll 1
    for (int sweep = 0; sweep < 60; sweep++) {
        bool changed = false;
#pragma unroll
        for (int i = 0; i < 7; i++) {
#pragma unroll
            for (int j = i + 1; j < 8; j++) {
                const float p = dot8(c[i], c[j]), ni = dot8(c[i], c[i]), nj = dot8(c[j], c[j]);
                // inner products below 1e-15 count as 0, so that columns of rounding noise end too
                if (p * p > fmaxf(eps2 * ni * nj, 1e-30f)) {
                    const float zeta = (nj - ni) / (2.0f * p), az = fabsf(zeta);
                    // tan(theta): smaller root of t^2 + 2 zeta t - 1 = 0 (1 / (2 zeta) once zeta^2 overflows)
                    const float t = copysignf(1.0f, zeta) / (az < 1e18f ? az + sqrtf(fmaf(zeta, zeta, 1.0f)) : 2.0f * az);
                    const float cs = 1.0f / sqrtf(fmaf(t, t, 1.0f)), sn = cs * t;
#pragma unroll
                    for (int k = 0; k < 4; k++) {
                        const float2 xi = c[i][k], xj = c[j][k];
                        c[i][k] = iqm::fma2(iqm::dup2(cs), xi, iqm::mul2(iqm::dup2(-sn), xj));
                        c[j][k] = iqm::fma2(iqm::dup2(sn), xi, iqm::mul2(iqm::dup2(cs), xj));
                    }
                    changed = true;
                }
            }
        }
        if (!changed) break;
    }
#pragma unroll
    for (int i = 0; i < 8; i++) {
        double q = 0.0;
#pragma unroll
        for (int k = 0; k < 4; k++) {
            q = fma(double(c[i][k].x), double(c[i][k].x), q);
            q = fma(double(c[i][k].y), double(c[i][k].y), q);
        }
        s[i] = float(sqrt(q));
    }
}

// Out of line and from the pixels again, so that this rare path holds no registers of the usual one.
__device__ __noinline__ void block_values_jacobi(const MsvdPairDev *pairs, int npairs, int slot, int img, float *out) {
    const MsvdPairDev P = pairs[find_pair(pairs, npairs, slot)];
    const int local = slot - P.slot_base;
    float2 c[8][4];
    float s[8];
    load_block(img ? P.b : P.a, P.pitch, 8 * (local % P.bw), 8 * (local / P.bw), P.vec_ok, c);
    svd8_jacobi(c, s);
#pragma unroll
    for (int i = 0; i < 8; i++) out[i] = s[i];
}

// Singular values (descending) of the 8x8 grey block of a slot and image; P is the slot's pair.
// Over 31 kinds of blocks (noise, text, edges, patches and sparse pixels on black and on white, flat and
// nearly flat, diagonal and block diagonal ones, of rank one and two; a million each) no value is 7.2e-4 away
// from its double-precision one, RMS 5e-5 and less (values up to 2040); one-sided Jacobi alone reaches 1.5e-3,
// RMS 1.3e-4, in more than twice the time, six to eight sweeps of 28 rotations.
__device__ __forceinline__ void block_values(const MsvdArgs &args, const MsvdPairDev &P, int bx, int by, int slot, int img,
                                             float (&s)[8]) {
    bool converged;
    {
        float2 c[8][4];
        load_block(img ? P.b : P.a, P.pitch, 8 * bx, 8 * by, P.vec_ok, c);
        converged = svd8_qd(c, s);
    }
    if (!converged) {
        float t[8];
        block_values_jacobi(args.pairs, args.npairs, slot, img, t);
#pragma unroll
        for (int i = 0; i < 8; i++) s[i] = t[i];
    }
    // descending order (sorting network on 8 registers)
#define IQM_CSWAP(a, b)                         \
    do {                                        \
        const float hi_ = fmaxf(s[a], s[b]);    \
        const float lo_ = fminf(s[a], s[b]);    \
        s[a] = hi_;                             \
        s[b] = lo_;                             \
    } while (0)
    IQM_CSWAP(0, 1); IQM_CSWAP(2, 3); IQM_CSWAP(4, 5); IQM_CSWAP(6, 7);
    IQM_CSWAP(0, 2); IQM_CSWAP(1, 3); IQM_CSWAP(4, 6); IQM_CSWAP(5, 7);
    IQM_CSWAP(1, 2); IQM_CSWAP(5, 6); IQM_CSWAP(0, 4); IQM_CSWAP(3, 7);
    IQM_CSWAP(1, 5); IQM_CSWAP(2, 6);
    IQM_CSWAP(1, 4); IQM_CSWAP(3, 6);
    IQM_CSWAP(2, 4); IQM_CSWAP(3, 5);
    IQM_CSWAP(3, 4);
#undef IQM_CSWAP
}

// Two lanes per block slot: the even lane takes the block of the distorted image, the odd lane the
// same block of the reference; the odd lane's singular values reach the even lane by shuffle.  One
// copy of the SVD code serves both images and twice as many blocks are in flight.
// Bound by instruction issue (78% of the issue slots, FMA pipe 54%, 5.0k instructions a warp of 16 blocks of both
// images, some of them lost to lanes that wait for their warp's slowest qd sweep).  16 1080p
// pairs: 475 us with Jacobi sweeps, 183 us now; five CTAs per SM at 93 registers took 185 us where six at 80
// took 178 us.
__global__ void __launch_bounds__(BLOCK_THREADS, 6) msvd_block_kernel(MsvdArgs args) {
    const int slot = (blockIdx.x * BLOCK_THREADS + threadIdx.x) >> 1;
    const int img = threadIdx.x & 1;
    const bool in_range = slot < args.total_slots;  // both lanes of a slot agree
    bool computed = false;
    MsvdPairDev P{};
    int bx = 0, by = 0;
    if (in_range) {
        P = args.pairs[find_pair(args.pairs, args.npairs, slot)];
        const int local = slot - P.slot_base;
        bx = local % P.bw;
        by = local / P.bw;
        computed = bx < P.vx && by < P.vy;  // other slots stay 0 (src/gpu/svd/svd.cpp:44,68-74)
    }
    // lanes that compute, fixed before the data-dependent sweeps (pairs of lanes agree)
    const unsigned mask = __ballot_sync(0xffffffffu, computed);
    if (computed) {
        {  // one 8x8 block of one image
            float s[8];
            block_values(args, P, bx, by, slot, img, s);
            float acc = 0.0f;  // shaders/svd/svd.glsl:41-52: float, k = 0..7 in order
#pragma unroll
            for (int k = 0; k < 8; k++) {
                const float sr = __shfl_xor_sync(mask, s[k], 1);
                const float t = s[k] - sr;
                acc = fmaf(t, t, acc);
            }
            if (!img) args.dist[slot] = sqrtf(acc);
        }
    }
    if (in_range && !computed && !img) args.dist[slot] = 0.0f;
}

__global__ void __launch_bounds__(POOL_THREADS) msvd_pool_kernel(MsvdArgs args) {
    __shared__ unsigned hist[iqm::SELECT_BINS];
    __shared__ double red_s[POOL_THREADS / 32];
    __shared__ float red_m[POOL_THREADS / 32];
    const MsvdPairDev &P = args.pairs[blockIdx.x];
    const int n = P.bw * P.bh;
    const float *D = args.dist + P.slot_base;
    const float med = iqm::block_select_kth(D, n, n / 2, hist);
    double s = 0.0;
    float mx = 0.0f;
    for (int i = threadIdx.x; i < n; i += POOL_THREADS) {
        const float v = __ldcg(D + i);
        s += double(fabsf(v - med));
        mx = fmaxf(mx, v);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        s += __shfl_down_sync(0xffffffffu, s, o);
        mx = fmaxf(mx, __shfl_down_sync(0xffffffffu, mx, o));
    }
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    if (lane == 0) {
        red_s[wid] = s;
        red_m[wid] = mx;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        float m = 0.0f;
        for (int w = 0; w < POOL_THREADS / 32; w++) {
            t += red_s[w];
            m = fmaxf(m, red_m[w]);
        }
        args.scores[blockIdx.x] = t / double(n);
        red_m[0] = m;
    }
    __syncthreads();
    if (P.map) {
        const float m = red_m[0];
        for (int i = threadIdx.x; i < n; i += POOL_THREADS) P.map[i] = __ldcg(D + i) / m;
    }
}

void msvd_enqueue(iqm_ctx *ctx, const std::vector<iqm_pair> &pairs, const std::vector<float *> &maps,
                  double *d_scores) {
    const int n = int(pairs.size());
    std::vector<MsvdPairDev> hd(n);
    long total = 0;
    for (int i = 0; i < n; i++) {
        const iqm_pair &q = pairs[i];
        MsvdPairDev &d = hd[i];
        d.a = q.input;
        d.b = q.ref;
        d.map = maps.empty() ? nullptr : maps[i];
        d.pitch = (long long)q.row_bytes;
        d.w = q.w;
        d.h = q.h;
        d.bw = q.w / 8;
        d.bh = q.h / 8;
        d.vx = q.w >= 9 ? (q.w - 1) / 8 : 0;  // x = 8*bx with x + 8 < W
        d.vy = q.h >= 9 ? (q.h - 1) / 8 : 0;
        d.slot_base = int(total);
        d.vec_ok = ((reinterpret_cast<uintptr_t>(q.input) | reinterpret_cast<uintptr_t>(q.ref) |
                     uintptr_t(q.row_bytes)) & 15u) == 0;
        total += long(d.bw) * d.bh;
    }
    IQM_REQUIRE(total < (1L << 31), "too many blocks in one batch");
    auto *d_desc = static_cast<MsvdPairDev *>(iqm::upload_bytes(ctx, ctx->desc, hd.data(), sizeof(MsvdPairDev) * n));
    MsvdArgs a{};
    a.pairs = d_desc;
    a.npairs = n;
    a.total_slots = int(total);
    a.dist = static_cast<float *>(ctx->scratch.get(sizeof(float) * size_t(total), ctx->stream));
    a.scores = d_scores;
    msvd_block_kernel<<<iqm::ceil_div(2 * total, BLOCK_THREADS), BLOCK_THREADS, 0, ctx->stream>>>(a);
    iqm::check_launch(ctx, "msvd_block_kernel");
    msvd_pool_kernel<<<n, POOL_THREADS, 0, ctx->stream>>>(a);
    iqm::check_launch(ctx, "msvd_pool_kernel");
}

}  // namespace

// The reference needs at least one 8x8 block slot: n = (W/8)*(H/8) > 0 (it divides by n).
static void check_msvd_pairs(const iqm_pair *pairs, int n) { iqm::check_pairs(pairs, n, 8, 8); }

void iqm::enqueue_msvd_dev(iqm_ctx *ctx, const iqm_pair *pairs, int n, double *d_scores) {
    check_msvd_pairs(pairs, n);
    iqm::check_dev_alignment(pairs, n);
    IQM_REQUIRE(d_scores != nullptr, "d_scores is NULL");
    msvd_enqueue(ctx, std::vector<iqm_pair>(pairs, pairs + n), {}, d_scores);
}

extern "C" __attribute__((visibility("default"))) int iqm_msvd_dev(iqm_ctx *ctx, const iqm_pair *pairs, int n,
                                                                  double *d_scores) {
    return iqm::guarded(ctx, [&] { iqm::enqueue_msvd_dev(ctx, pairs, n, d_scores); });
}

extern "C" __attribute__((visibility("default"))) int iqm_msvd_batch(iqm_ctx *ctx, const iqm_pair *pairs, int n,
                                                                    double *scores) {
    return iqm::guarded(ctx, [&] {
        check_msvd_pairs(pairs, n);
        IQM_REQUIRE(scores != nullptr, "scores is NULL");
        auto *d_scores = static_cast<double *>(ctx->scores.get(sizeof(double) * n, ctx->stream));
        iqm::upload_pipelined(ctx, pairs, n, [&](const iqm_pair *dev, int first, int count) {
            msvd_enqueue(ctx, std::vector<iqm_pair>(dev, dev + count), {}, d_scores + first);
        });
        IQM_CHECK_CUDA(cudaMemcpyAsync(scores, d_scores, sizeof(double) * n, cudaMemcpyDeviceToHost, ctx->stream));
        IQM_CHECK_CUDA(cudaStreamSynchronize(ctx->stream));
    });
}

extern "C" __attribute__((visibility("default"))) int iqm_msvd(iqm_ctx *ctx, const uint8_t *rgba_in,
                                                              const uint8_t *rgba_ref, int w, int h,
                                                              size_t row_bytes, float *block_map, double *msvd) {
    return iqm::guarded(ctx, [&] {
        IQM_REQUIRE(msvd != nullptr, "msvd is NULL");
        iqm_pair hp{rgba_in, rgba_ref, w, h, row_bytes};
        check_msvd_pairs(&hp, 1);
        auto dev = iqm::upload_pairs(ctx, &hp, 1);
        auto *d_score = static_cast<double *>(ctx->scores.get(sizeof(double), ctx->stream));
        const size_t nb = size_t(w / 8) * size_t(h / 8);
        std::vector<float *> maps;
        float *d_map = nullptr;
        if (block_map) {
            d_map = static_cast<float *>(ctx->maps.get(sizeof(float) * nb, ctx->stream));
            maps.push_back(d_map);
        }
        msvd_enqueue(ctx, dev, maps, d_score);
        IQM_CHECK_CUDA(cudaMemcpyAsync(msvd, d_score, sizeof(double), cudaMemcpyDeviceToHost, ctx->stream));
        if (block_map)
            IQM_CHECK_CUDA(cudaMemcpyAsync(block_map, d_map, sizeof(float) * nb, cudaMemcpyDeviceToHost, ctx->stream));
        IQM_CHECK_CUDA(cudaStreamSynchronize(ctx->stream));
    });
}
