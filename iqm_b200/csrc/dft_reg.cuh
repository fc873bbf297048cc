// DFTs of 2 to 32 points held in one thread's registers, sign +1: V_q = sum_r v_r exp(2 pi i r q / P).
//
// Sizes up to 15 with factors 2, 3 and 5 are fft.cuh's.  Here: odd primes (symmetric pairs, direct
// sums), coprime products (Good-Thomas, dft_pfa of fft.cuh) and prime powers (Cooley-Tukey with
// constant twiddles).  All coefficients are compile-time constants, so they become instruction
// immediates and a transform needs no registers beyond its points and temporaries.
#pragma once

#include "fft.cuh"

namespace iqm {

// cos and sin of 2 pi num / den, evaluated at compile time: the angle is reduced to [-pi, pi] and
// summed as its Taylor series (24 terms leave less than 1e-16).
__host__ __device__ constexpr double trig_angle(int num, int den) {
    int k = num % den;
    if (2 * k > den) k -= den;
    return 6.283185307179586476925286766559 * double(k) / double(den);
}
__host__ __device__ constexpr double cos_turn(int num, int den) {
    const double x = trig_angle(num, den), x2 = x * x;
    double term = 1.0, sum = 1.0;
    for (int i = 1; i <= 24; i++) {
        term *= -x2 / double((2 * i - 1) * (2 * i));
        sum += term;
    }
    return sum;
}
__host__ __device__ constexpr double sin_turn(int num, int den) {
    const double x = trig_angle(num, den), x2 = x * x;
    double term = x, sum = x;
    for (int i = 1; i <= 24; i++) {
        term *= -x2 / double((2 * i) * (2 * i + 1));
        sum += term;
    }
    return sum;
}

// The constants as static data members, so they are evaluated at compile time wherever they are used.
template <int K, int N>
struct Turn {
    static constexpr float c = float(cos_turn(K, N)), s = float(sin_turn(K, N));
};

// Calls f(integral constant I) for I = B .. E - 1.
template <int B, int E, class F>
__device__ __forceinline__ void static_for(F &&f) {
    if constexpr (B < E) {
        f(std::integral_constant<int, B>{});
        static_for<B + 1, E>(static_cast<F &&>(f));
    }
}

// Odd prime P: with a_r = v_r + v_{P-r}, b_r = v_r - v_{P-r}, X_q and X_{P-q} are
// v_0 + sum_r a_r cos(2 pi r q / P) +- i sum_r b_r sin(2 pi r q / P).
template <int P>
__device__ __forceinline__ void dft_prime(float2 *v) {
    constexpr int H = (P - 1) / 2;
    float2 a[H], b[H];
    float2 sum = v[0];
#pragma unroll
    for (int r = 0; r < H; r++) {
        a[r] = cadd(v[r + 1], v[P - 1 - r]);
        b[r] = csub(v[r + 1], v[P - 1 - r]);
        sum = cadd(sum, a[r]);
    }
    const float2 x0 = v[0];
    v[0] = sum;
    static_for<1, H + 1>([&](auto Q) {
        constexpr int q = decltype(Q)::value;
        float2 re = x0, im = make_float2(0.f, 0.f);
        static_for<1, H + 1>([&](auto R) {
            constexpr int r = decltype(R)::value;
            constexpr float c = Turn<(r * q) % P, P>::c, s = Turn<(r * q) % P, P>::s;
            re.x = fmaf(a[r - 1].x, c, re.x);
            re.y = fmaf(a[r - 1].y, c, re.y);
            im.x = fmaf(b[r - 1].x, s, im.x);
            im.y = fmaf(b[r - 1].y, s, im.y);
        });
        v[q] = make_float2(re.x - im.y, re.y + im.x);
        v[P - q] = make_float2(re.x + im.y, re.y - im.x);
    });
}

template <int P>
__device__ __forceinline__ void dft_reg(float2 *v);

// P = N1 N2 (Cooley-Tukey): n = N2 n1 + n2, k = k1 + N1 k2.
template <int N1, int N2>
__device__ __forceinline__ void dft_ct(float2 *v) {
    constexpr int N = N1 * N2;
    float2 t[N2][N1];
    static_for<0, N2>([&](auto I) {
        constexpr int n2 = decltype(I)::value;
#pragma unroll
        for (int n1 = 0; n1 < N1; n1++) t[n2][n1] = v[N2 * n1 + n2];
        dft_reg<N1>(t[n2]);
        static_for<1, N1>([&](auto K) {
            constexpr int k1 = decltype(K)::value;
            constexpr int e = (n2 * k1) % N;
            if constexpr (e != 0) {
                const float2 u = t[n2][k1];
                if constexpr (4 * e == N)
                    t[n2][k1] = make_float2(-u.y, u.x);
                else if constexpr (2 * e == N)
                    t[n2][k1] = make_float2(-u.x, -u.y);
                else if constexpr (4 * e == 3 * N)
                    t[n2][k1] = make_float2(u.y, -u.x);
                else
                    t[n2][k1] = make_float2(u.x * Turn<e, N>::c - u.y * Turn<e, N>::s,
                                            u.x * Turn<e, N>::s + u.y * Turn<e, N>::c);
            }
        });
    });
#pragma unroll
    for (int k1 = 0; k1 < N1; k1++) {
        float2 b[N2];
#pragma unroll
        for (int n2 = 0; n2 < N2; n2++) b[n2] = t[n2][k1];
        dft_reg<N2>(b);
#pragma unroll
        for (int k2 = 0; k2 < N2; k2++) v[k1 + N1 * k2] = b[k2];
    }
}

// Good-Thomas product of coprime sizes without twiddles (the mapping of fft.cuh's dft_pfa).
template <int N1, int N2>
__device__ __forceinline__ void dft_gt(float2 *v) {
    constexpr int N = N1 * N2;
    constexpr int A = mod_inverse(N2 % N1, N1), B = mod_inverse(N1 % N2, N2);
    float2 t[N2][N1];
#pragma unroll
    for (int n2 = 0; n2 < N2; n2++) {
#pragma unroll
        for (int n1 = 0; n1 < N1; n1++) t[n2][n1] = v[(n1 * N2 + n2 * N1) % N];
        dft_reg<N1>(t[n2]);
    }
#pragma unroll
    for (int k1 = 0; k1 < N1; k1++) {
        float2 b[N2];
#pragma unroll
        for (int n2 = 0; n2 < N2; n2++) b[n2] = t[n2][k1];
        dft_reg<N2>(b);
#pragma unroll
        for (int k2 = 0; k2 < N2; k2++) v[(k1 * N2 * A + k2 * N1 * B) % N] = b[k2];
    }
}

template <int P>
__device__ __forceinline__ void dft_reg(float2 *v) {
    if constexpr (P == 1) {
    } else if constexpr (P == 2 || P == 3 || P == 4 || P == 5 || P == 6 || P == 8 || P == 9 || P == 10 || P == 12 || P == 15) {
        dft_small<P>(v, 1.f);
    } else if constexpr (P == 16) {
        dft_ct<4, 4>(v);
    } else if constexpr (P == 25) {
        dft_ct<5, 5>(v);
    } else if constexpr (P == 27) {
        dft_ct<3, 9>(v);
    } else if constexpr (P == 32) {
        dft_ct<4, 8>(v);
    } else if constexpr (P == 24) {
        dft_gt<3, 8>(v);
    } else if constexpr (P == 20 || P == 28) {
        dft_gt<4, P / 4>(v);
    } else if constexpr (P == 21) {
        dft_gt<3, 7>(v);
    } else if constexpr (P % 2 == 0) {  // 14, 18, 22, 26, 30
        dft_gt<2, P / 2>(v);
    } else {
        dft_prime<P>(v);
    }
}

}  // namespace iqm
