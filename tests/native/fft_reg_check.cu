// The register FFT engine's plans (fft_reg.cu) followed step by step on the host: for every length in
// [argv 1, argv 2], each step's radix is one its kernels implement, its lines cover the matrix exactly
// once within the sequence's shared memory, and the steps together with their tables compute the DFT.
// Prints "<n> <kind> <error>" per length (error relative to the inputs' norm), or a line starting BAD.
#include <cmath>
#include <complex>
#include <cstdio>
#include <cstdlib>
#include <vector>

#include "fft_reg_plan.cuh"

using Z = std::complex<double>;

static int div_host(int i, float inv) { return int((float(i) + 0.5f) * inv); }
static Z z(float2 v) { return Z(v.x, v.y); }

static void dft(std::vector<Z> &v) {
    const long p = long(v.size());
    std::vector<Z> out(p);
    for (long q = 0; q < p; q++)
        for (long r = 0; r < p; r++) out[q] += v[r] * std::polar(1.0, 2.0 * M_PI * double(r * q % p) / double(p));
    v = out;
}

static bool check(int n) {
    iqm::RegFft F;
    int kind = -1;
    if (!iqm::reg_plan(n, F, kind)) return std::printf("%d none 0\n", n), true;
    iqm::RegTables T;
    iqm::reg_tables(F, T);
    std::vector<Z> x(n), out(n), sm(F.size);
    double norm = 0.0;
    for (Z &v : x) v = Z(drand48() - 0.5, drand48() - 0.5), norm += std::norm(v);
    for (int k = 0; k < F.nsteps; k++) {
        const iqm::RegStep &S = F.st[k];
        const bool last = k == F.nsteps - 1, any_radix = k == 0 && !(kind == iqm::REG_THREE && F.blue);
        if (!iqm::reg_radix_ok(kind, any_radix ? 0 : 1, S.radix)) return std::printf("BAD radix %d\n", n), false;
        if (S.items * S.radix != F.m || (S.tw < 0) != last) return std::printf("BAD step %d\n", n), false;
        std::vector<char> seen(F.size, 0);
        for (int i = 0; i < S.items; i++) {
            const int q = div_host(i, S.inv_d0), base = q * S.hi + (i - q * S.d0) * S.lo;
            if (q != i / S.d0) return std::printf("BAD quotient %d\n", n), false;
            std::vector<Z> v(S.radix);
            for (int r = 0; r < S.radix; r++) {
                const int a = base + r * S.stride, e = i + r * S.items;
                if (a < 0 || a >= F.size || seen[a]++) return std::printf("BAD address %d\n", n), false;
                if (k == 0) v[r] = e < n ? (F.blue ? x[e] * z(T.data[T.chirp + e]) : x[e]) : Z(0.0);
                else v[r] = sm[a];
            }
            dft(v);
            if (F.blue && k == F.fused) {
                for (int r = 0; r < S.radix; r++) {
                    const Z t = v[r] * z(T.data[T.bhat + i + r * S.items]);
                    v[r] = Z(t.imag(), t.real());
                }
                dft(v);
            }
            for (int r = 0; r < S.radix; r++) {
                const int a = base + r * S.stride, e = i + r * S.items;
                if (!last) {
                    sm[a] = v[r] * z(T.data[S.tw + e]);
                } else if (e < n) {
                    out[e] = F.blue ? Z(v[r].imag(), v[r].real()) * z(T.data[T.chirp + e]) : v[r];
                    const int rr = div_host(e, F.inv_items_last), ii = e - rr * S.items, qq = div_host(ii, S.inv_d0);
                    if (qq * S.hi + (ii - qq * S.d0) * S.lo + rr * S.stride != a) return std::printf("BAD place %d\n", n), false;
                }
            }
        }
    }
    double err = 0.0;
    for (int k : {0, 1 % n, n / 3, n - 1}) {
        Z want = 0.0;
        for (long t = 0; t < n; t++) want += x[t] * std::polar(1.0, 2.0 * M_PI * double(t * k % n) / double(n));
        err = std::fmax(err, std::abs(want - out[k]));
    }
    std::printf("%d %d %.3e\n", n, kind, err / std::sqrt(norm));
    return true;
}

int main(int argc, char **argv) {
    if (argc != 3) return 2;
    for (int n = std::atoi(argv[1]); n <= std::atoi(argv[2]); n++)
        if (!check(n)) return 1;
    return 0;
}
