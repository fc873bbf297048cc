// Complex FP32 FFTs of whole sequences by a CTA, most of the work in registers (sm_100a).
//
// A length m = p1 p2 (p3) is a matrix in shared memory, element n = (n1 p2 + n2) p3 + n3 at address
// n1 s1 + n2 s2 + n3.  Every step is a DFT along one axis: a thread takes one line of the axis (up to
// 32 points) into registers (dft_reg.cuh), transforms it, multiplies by the step's twiddles and writes
// it back to the same places, so the transform is in place, a step's lines are independent, and one
// barrier separates steps.  The first step reads its lines straight from the caller's source and the
// last one hands them to the caller's sink, so a two-factor transform crosses shared memory once.
// Output k = k1 + p1 (k2 + p2 k3) sits where element (k1, k2, k3) does.
//
// Lengths without such factors run through Bluestein's chirp-z algorithm on m >= 2n - 1.  The forward
// transform's last axis is also the inverse transform's first one, so one step transforms a line,
// multiplies it by the kernel's spectrum and transforms it back without leaving the registers: a
// two-factor Bluestein transform is three steps and crosses shared memory twice.
//
// All transforms have sign +1; sign -1 is the same transform with real and imaginary parts exchanged
// on the way in and out (which is also how Bluestein's inner inverse runs).
//
// In every step line i of `items` holds the logical elements i + r items, r < radix; the twiddle
// tables, Bluestein's kernel, inputs and outputs are all indexed by that number, so neighbouring
// lines read neighbouring entries.
#pragma once

#include <type_traits>

#include "dft_reg.cuh"

namespace iqm {

constexpr int REG_MAX_STEPS = 5;

struct RegStep {
    int radix;
    int items;    // lines of the axis: m / radix
    int d0;       // line i starts at (i / d0) hi + (i % d0) lo
    float inv_d0;
    int hi, lo;
    int stride;   // between the points of a line
    int tw;       // offset of the step's twiddles in RegFft::tw (-1: none)
    float inv_items;
};

struct RegFft {
    int n;        // transform length
    int m;        // matrix points: n, or Bluestein's length
    int blue;     // Bluestein
    int nsteps;
    int fused;    // index of the Bluestein step that transforms forth and back
    int size;     // shared-memory points per sequence
    int stages;   // factors of m (2 or 3)
    int max_radix;
    float inv_items_last;  // 1 / items of the last step
    RegStep st[REG_MAX_STEPS];
    const float2 *tw;     // per step [r][line]
    const float2 *chirp;  // exp(+pi i t^2 / n), t < n
    const float2 *bhat;   // transform of the wrapped conjugate chirp, divided by m
};

// Shared memory by 32-bit byte address, so that stepping along a line costs one integer instruction a
// point.
__device__ __forceinline__ unsigned smem_addr(const void *p) { return static_cast<unsigned>(__cvta_generic_to_shared(p)); }
__device__ __forceinline__ float2 lds2(unsigned a) {
    float2 v;
    asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ float lds1(unsigned a) {
    float v;
    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ void sts2(unsigned a, float2 v) {
    asm volatile("st.shared.v2.f32 [%0], {%1, %2};" ::"r"(a), "f"(v.x), "f"(v.y) : "memory");
}
// Element r of a strided run in global memory: one wide multiply-add forms the address.
template <class T>
__device__ __forceinline__ const T *run_at(const T *first, unsigned byte_stride, unsigned r) {
    return reinterpret_cast<const T *>(reinterpret_cast<const char *>(first) + static_cast<unsigned long long>(byte_stride) * r);
}
template <class T>
__device__ __forceinline__ T *run_at(T *first, unsigned byte_stride, unsigned r) {
    return reinterpret_cast<T *>(reinterpret_cast<char *>(first) + static_cast<unsigned long long>(byte_stride) * r);
}

// i / d for 0 <= i < 2^22 with inv = 1 / d
__device__ __forceinline__ int div_by(int i, float inv) { return __float2int_rz((float(i) + 0.5f) * inv); }

// Where a CTA's sequences live.  Columns: C = 2^lc adjacent columns interleaved point by point (c
// fastest), so neighbouring threads take neighbouring columns.  Rows: one sequence after another.
template <int LC>  // log2 columns (-1: the member says)
struct ColLayout {
    int lc_;
    int count;  // columns in use (<= 2^lc)
    int threads;
    __device__ __forceinline__ int lc() const { return LC >= 0 ? LC : lc_; }
    __device__ __forceinline__ int first() const { return threadIdx.x; }
    __device__ __forceinline__ int total(int items) const { return items << lc(); }
    __device__ __forceinline__ void split(int w, const RegStep &, int &seq, int &i) const {
        seq = w & ((1 << lc()) - 1);
        i = w >> lc();
    }
    __device__ __forceinline__ bool live(int seq) const { return seq < count; }
    __device__ __forceinline__ int addr(int seq, int a) const { return (a << lc()) + seq; }
    __device__ __forceinline__ int stride(int s) const { return s << lc(); }
};
struct RowLayout {
    int count;
    int size;
    int threads;
    __device__ __forceinline__ int first() const { return threadIdx.x; }
    __device__ __forceinline__ int total(int items) const { return items * count; }
    __device__ __forceinline__ void split(int w, const RegStep &S, int &seq, int &i) const {
        seq = div_by(w, S.inv_items);
        i = w - seq * S.items;
    }
    __device__ __forceinline__ bool live(int) const { return true; }
    __device__ __forceinline__ int addr(int seq, int a) const { return seq * size + a; }
    __device__ __forceinline__ int stride(int s) const { return s; }
};

__device__ __forceinline__ int line_base(const RegStep &S, int i) {
    const int q = div_by(i, S.inv_d0);
    return q * S.hi + (i - q * S.d0) * S.lo;
}

// Multiplies points r >= R0 of line i by the step's twiddles.
template <int P, int R0>
__device__ __forceinline__ void twiddle_line(float2 *v, const RegFft &F, const RegStep &S, int i) {
    const float2 *tw = F.tw + S.tw + i;
    const unsigned d = unsigned(S.items) * 8u;
#pragma unroll
    for (int r = R0; r < P; r++) v[r] = cmul(v[r], __ldg(run_at(tw, d, r)));
}

// Points of line i that are inputs or outputs of a Bluestein transform, i + r items < n: fewer than half the
// line and one, as n <= (m + 1) / 2, so the rest of the line is left out at compile time.
template <int P>
constexpr int kHalf = (P + 2) / 2;
__device__ __forceinline__ int live_points(const RegFft &F, const RegStep &S, int i) {
    return div_by(F.n - i + S.items - 1, S.inv_items);
}

// First step: ld(seq, i, items)(r), element i + r items of a sequence -> lines -> shared memory.
template <int P, bool BLUE, class Lay, class Ld>
__device__ __forceinline__ void reg_first(const RegFft &F, const Lay &lay, float2 *sm, Ld &ld) {
    const RegStep &S = F.st[0];
    const int total = lay.total(S.items);
    for (int w = lay.first(); w < total; w += lay.threads) {
        int seq, i;
        lay.split(w, S, seq, i);
        if (!lay.live(seq)) continue;
        auto src = ld(seq, i, S.items);
        float2 v[P];
        if constexpr (BLUE) {
            const int live = live_points(F, S, i);
#pragma unroll
            for (int r = 0; r < P; r++) v[r] = r < kHalf<P> && r < live ? src(r) : make_float2(0.f, 0.f);
            const float2 *chirp = F.chirp + i;
#pragma unroll
            for (int r = 0; r < kHalf<P>; r++)
                if (r < live) v[r] = cmul(v[r], __ldg(run_at(chirp, 8u * S.items, r)));
        } else {
#pragma unroll
            for (int r = 0; r < P; r++) v[r] = src(r);
        }
        dft_reg<P>(v);
        twiddle_line<P, 1>(v, F, S, i);
        const unsigned p = smem_addr(sm) + 8u * lay.addr(seq, line_base(S, i)), d = 8u * lay.stride(S.stride);
#pragma unroll
        for (int r = 0; r < P; r++) sts2(p + r * d, v[r]);
    }
}

// UNIT: the step's lines are runs of neighbouring points (the last axis), so that every point of a line
// is at a constant offset.
// Middle step, in place: a DFT and the step's twiddles; FUSED: forth, times Bluestein's kernel, and back
// (the back transform's exchange of parts is undone by the last step).
template <int P, bool FUSED, bool UNIT, class Lay>
__device__ __forceinline__ void reg_middle(const RegFft &F, const RegStep &S, const Lay &lay, float2 *sm) {
    const int total = lay.total(S.items);
    for (int w = lay.first(); w < total; w += lay.threads) {
        int seq, i;
        lay.split(w, S, seq, i);
        if (!lay.live(seq)) continue;
        const unsigned p = smem_addr(sm) + 8u * lay.addr(seq, line_base(S, i)), d = 8u * lay.stride(UNIT ? 1 : S.stride);
        float2 v[P];
#pragma unroll
        for (int r = 0; r < P; r++) v[r] = lds2(p + r * d);
        dft_reg<P>(v);
        if constexpr (FUSED) {
#pragma unroll
            for (int r = 0; r < P; r++) {
                const float2 t = cmul(v[r], __ldg(run_at(F.bhat + i, 8u * S.items, r)));
                v[r] = make_float2(t.y, t.x);
            }
            dft_reg<P>(v);
        }
        twiddle_line<P, 0>(v, F, S, i);
#pragma unroll
        for (int r = 0; r < P; r++) sts2(p + r * d, v[r]);
    }
}

// Last step: lines -> st(seq, i, items)(r, place, value).
template <int P, bool BLUE, bool UNIT, class Lay, class St>
__device__ __forceinline__ void reg_last(const RegFft &F, const RegStep &S, const Lay &lay, float2 *sm, St &st) {
    const int total = lay.total(S.items);
    for (int w = lay.first(); w < total; w += lay.threads) {
        int seq, i;
        lay.split(w, S, seq, i);
        if (!lay.live(seq)) continue;
        const unsigned p = smem_addr(sm) + 8u * lay.addr(seq, line_base(S, i)), d = 8u * lay.stride(UNIT ? 1 : S.stride);
        float2 v[P];
#pragma unroll
        for (int r = 0; r < P; r++) v[r] = lds2(p + r * d);
        dft_reg<P>(v);
        auto dst = st(seq, i, S.items);
        if constexpr (BLUE) {
            const int live = live_points(F, S, i);
            const float2 *chirp = F.chirp + i;
#pragma unroll
            for (int r = 0; r < kHalf<P>; r++)
                if (r < live) dst(r, p + r * d, cmul(make_float2(v[r].y, v[r].x), __ldg(run_at(chirp, 8u * S.items, r))));
        } else {
#pragma unroll
            for (int r = 0; r < P; r++) dst(r, p + r * d, v[r]);
        }
    }
}

// Kinds of plan a kernel is compiled for, so that each holds the code and registers of its own radices.
enum RegKind { REG_DIRECT_24 = 0, REG_DIRECT_32 = 1, REG_BLUE_2 = 2, REG_THREE = 3, REG_BLUE_24 = 4, REG_KINDS = 5 };

// Radices the steps of each kind implement.  First steps take any radix up to the kind's largest; the
// others leave out the larger primes, which a plan puts first.
__host__ __device__ constexpr bool reg_radix_ok(int kind, int where /* 0 first, 1 middle or last */, int p) {
    const bool smooth = p == 8 || p == 9 || p == 10 || p == 12 || p == 15 || p == 16 || p == 18 || p == 20;
    const bool small = p >= 4 && p <= 7;
    switch (kind) {
        case REG_DIRECT_24:
            return where == 0 ? p >= 2 && p <= 24
                              : p >= 1 && p <= 24 && p != 17 && p != 19 && p != 23;
        case REG_DIRECT_32:
            return where == 0 ? p >= 2 && p <= 32
                              : p >= 7 && p <= 32 && p != 17 && p != 19 && p != 23 && p != 29 && p != 31;
        case REG_BLUE_2:
            return smooth || p == 24 || p == 25 || p == 27 || p == 28 || p == 30 || p == 32;
        case REG_BLUE_24:
            return smooth || p == 24;
        default:
            return where == 0 ? p >= 2 && p <= 20 : smooth || small;
    }
}

template <int KIND, int WHERE, class F>
__device__ __forceinline__ void with_radix(int radix, F &&f) {
#define IQM_RADIX(P)                                                       \
    case P:                                                                \
        if constexpr (reg_radix_ok(KIND, WHERE, P)) f(std::integral_constant<int, P>{}); \
        break;
    switch (radix) {
        IQM_RADIX(1) IQM_RADIX(2) IQM_RADIX(3) IQM_RADIX(4) IQM_RADIX(5) IQM_RADIX(6) IQM_RADIX(7) IQM_RADIX(8)
        IQM_RADIX(9) IQM_RADIX(10) IQM_RADIX(11) IQM_RADIX(12) IQM_RADIX(13) IQM_RADIX(14) IQM_RADIX(15) IQM_RADIX(16)
        IQM_RADIX(17) IQM_RADIX(18) IQM_RADIX(19) IQM_RADIX(20) IQM_RADIX(21) IQM_RADIX(22) IQM_RADIX(23) IQM_RADIX(24)
        IQM_RADIX(25) IQM_RADIX(26) IQM_RADIX(27) IQM_RADIX(28) IQM_RADIX(29) IQM_RADIX(30) IQM_RADIX(31) IQM_RADIX(32)
        default: break;
    }
#undef IQM_RADIX
}

// The whole transform of the CTA's sequences; every thread of the CTA calls it.  ld(seq, i,
// items) and st(seq, i, items) give functions for one line: of r, its input i + r items, and of (r, place,
// value), which takes output i + r items (`place`: the byte address of its own slot in
// shared memory, whose old value no thread needs any more).  The caller puts a barrier before `sm` is used again.
template <int KIND, class Lay, class Ld, class St>
__device__ __forceinline__ void reg_fft(const RegFft &F, const Lay &lay, float2 *sm, Ld ld, St st) {
    if constexpr (KIND == REG_DIRECT_24 || KIND == REG_DIRECT_32) {
        with_radix<KIND, 0>(F.st[0].radix, [&](auto P) { reg_first<decltype(P)::value, false>(F, lay, sm, ld); });
        __syncthreads();
        with_radix<KIND, 1>(F.st[1].radix, [&](auto P) { reg_last<decltype(P)::value, false, true>(F, F.st[1], lay, sm, st); });
    } else if constexpr (KIND == REG_BLUE_2 || KIND == REG_BLUE_24) {
        with_radix<KIND, 0>(F.st[0].radix, [&](auto P) { reg_first<decltype(P)::value, true>(F, lay, sm, ld); });
        __syncthreads();
        with_radix<KIND, 1>(F.st[1].radix, [&](auto P) { reg_middle<decltype(P)::value, true, true>(F, F.st[1], lay, sm); });
        __syncthreads();
        with_radix<KIND, 1>(F.st[2].radix, [&](auto P) { reg_last<decltype(P)::value, true, false>(F, F.st[2], lay, sm, st); });
    } else if (!F.blue) {
        with_radix<KIND, 0>(F.st[0].radix, [&](auto P) { reg_first<decltype(P)::value, false>(F, lay, sm, ld); });
        __syncthreads();
        with_radix<KIND, 1>(F.st[1].radix, [&](auto P) { reg_middle<decltype(P)::value, false, false>(F, F.st[1], lay, sm); });
        __syncthreads();
        with_radix<KIND, 1>(F.st[2].radix, [&](auto P) { reg_last<decltype(P)::value, false, true>(F, F.st[2], lay, sm, st); });
    } else {
        with_radix<KIND, 1>(F.st[0].radix, [&](auto P) { reg_first<decltype(P)::value, true>(F, lay, sm, ld); });
        __syncthreads();
        with_radix<KIND, 1>(F.st[1].radix, [&](auto P) { reg_middle<decltype(P)::value, false, false>(F, F.st[1], lay, sm); });
        __syncthreads();
        with_radix<KIND, 1>(F.st[2].radix, [&](auto P) { reg_middle<decltype(P)::value, true, true>(F, F.st[2], lay, sm); });
        __syncthreads();
        with_radix<KIND, 1>(F.st[3].radix, [&](auto P) { reg_middle<decltype(P)::value, false, false>(F, F.st[3], lay, sm); });
        __syncthreads();
        with_radix<KIND, 1>(F.st[4].radix, [&](auto P) { reg_last<decltype(P)::value, true, false>(F, F.st[4], lay, sm, st); });
    }
}

// Where output k of a transform whose sink left it in place sits.
__device__ __forceinline__ int reg_out_addr(const RegFft &F, const RegStep &last, int k) {
    const int r = div_by(k, F.inv_items_last);
    return line_base(last, k - r * last.items) + r * last.stride;
}

}  // namespace iqm
