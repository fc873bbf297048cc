// Host side of the register FFT engine (fft_reg.cuh): the choice of factors and the device tables of a
// length, cached on the context.
#include <algorithm>
#include <cmath>
#include <complex>
#include <memory>
#include <vector>

#include "fft_reg_plan.cuh"
#include "iqm_internal.cuh"

namespace iqm {

struct RegPlan {
    RegFft fft{};
    int kind = -1;
    void *dev = nullptr;
    ~RegPlan() {
        if (dev) cudaFree(dev);
    }
};

namespace {

// Instructions of a P-point register DFT (additions are packed, so a complex one is one instruction).
int dft_cost(int p) {
    auto product = [](int a, int b, int twiddles) { return b * dft_cost(a) + a * dft_cost(b) + 4 * twiddles; };
    switch (p) {
        case 1: return 0;
        case 2: return 2;
        case 3: return 11;
        case 4: return 10;
        case 5: return 29;
        case 6: return product(2, 3, 0);
        case 8: return product(4, 2, 2);
        case 9: return product(3, 3, 4);
        case 10: return product(2, 5, 0);
        case 12: return product(4, 3, 0);
        case 15: return product(3, 5, 0);
        case 16: return product(4, 4, 8);
        case 20: return product(4, 5, 0);
        case 21: return product(3, 7, 0);
        case 24: return product(3, 8, 0);
        case 25: return product(5, 5, 16);
        case 27: return product(3, 9, 16);
        case 28: return product(4, 7, 0);
        case 32: return product(4, 8, 20);
        default: break;
    }
    if (p % 2 == 0) return product(2, p / 2, 0);
    const int h = (p - 1) / 2;
    return 4 * h * h + 6 * h;
}

// A step's line: the DFT, its loads, stores, twiddles and addresses, and the line's own index work.
int line_cost(int p) { return dft_cost(p) + 11 * p + 30; }

RegStep make_step(int radix, int items, int d0, int hi, int lo, int stride) {
    RegStep s{};
    s.radix = radix;
    s.items = items;
    s.d0 = d0;
    s.inv_d0 = 1.0f / float(d0);
    s.inv_items = 1.0f / float(items);
    s.hi = hi;
    s.lo = lo;
    s.stride = stride;
    s.tw = -1;
    return s;
}

// Lays out m = p1 p2 p3 (p3 = 1: two factors).  Odd strides between the lines of the later axes keep
// their shared-memory accesses free of bank conflicts.
RegFft build(int n, bool blue, int p1, int p2, int p3) {
    RegFft F{};
    F.n = n;
    F.m = p1 * p2 * p3;
    F.blue = blue ? 1 : 0;
    F.stages = p3 > 1 ? 3 : 2;
    F.max_radix = std::max(p1, std::max(p2, p3));
    const int s2 = p3 > 1 ? (p3 | 1) : 1;
    const int s1 = (p2 * s2) | 1;
    F.size = p1 * s1;
    const RegStep axis1 = make_step(p1, p2 * p3, p3, s2, 1, s1);
    const RegStep axis2 = p3 > 1 ? make_step(p2, p1 * p3, p3, s1, 1, s2) : make_step(p2, p1, p1, 0, s1, 1);
    const RegStep axis3 = make_step(p3, p1 * p2, p1, s2, s1, 1);
    int k = 0, off = 0;
    auto add = [&](RegStep s, bool twiddles) {
        if (twiddles) {
            s.tw = off;
            off += F.m;
        }
        F.st[k++] = s;
    };
    add(axis1, true);
    if (p3 > 1) {
        add(axis2, true);
        F.fused = 2;
        add(axis3, blue);
        if (blue) {
            add(axis2, true);
            add(axis1, false);
        }
    } else {
        F.fused = 1;
        add(axis2, blue);
        if (blue) add(axis1, false);
    }
    F.nsteps = k;
    F.inv_items_last = F.st[k - 1].inv_items;
    return F;
}

}  // namespace

long long reg_cost(const RegFft &F) {
    long long c = 0;
    for (int k = 0; k < F.nsteps; k++) {
        long long line = line_cost(F.st[k].radix);
        if (F.blue && k == F.fused) line += dft_cost(F.st[k].radix) + 8 * F.st[k].radix;
        c += line * F.st[k].items + 400;  // and a barrier's share
    }
    if (F.blue) c += 12LL * F.n;  // chirps
    return c;
}

bool reg_plan(int n, RegFft &best, int &kind) {
    if (n < 2) return false;
    long long best_cost = -1;
    auto consider = [&](bool blue, int p1, int p2, int p3, int k) {
        if ((long long)p1 * p2 * p3 > REG_MAX_POINTS) return;
        const RegFft F = build(n, blue, p1, p2, p3);
        // kernels of 80 registers a thread keep half as many warps more resident than those of 128
        const long long c = reg_cost(F) * (k == REG_DIRECT_32 || k == REG_BLUE_2 ? 5 : 4);
        if (best_cost < 0 || c < best_cost) {
            best_cost = c;
            best = F;
            kind = k;
        }
    };
    for (int p1 = 2; p1 <= 32; p1++) {
        for (int p2 = 1; p2 <= 32; p2++) {
            const int k = p1 <= 24 && p2 <= 24 ? REG_DIRECT_24 : REG_DIRECT_32;
            if (p1 * p2 == n && reg_radix_ok(k, 0, p1) && reg_radix_ok(k, 1, p2)) consider(false, p1, p2, 1, k);
            if (p1 * p2 >= 2 * n - 1) {
                const int kb = p1 <= 24 && p2 <= 24 ? REG_BLUE_24 : REG_BLUE_2;
                if (reg_radix_ok(kb, 1, p1) && reg_radix_ok(kb, 1, p2)) consider(true, p1, p2, 1, kb);
            }
            if (p1 > 20 || !reg_radix_ok(REG_THREE, 1, p2)) continue;
            for (int p3 = 4; p3 <= 20; p3++) {
                if (!reg_radix_ok(REG_THREE, 1, p3)) continue;
                if (p1 * p2 * p3 == n) consider(false, p1, p2, p3, REG_THREE);
                if (p1 * p2 * p3 >= 2 * n - 1 && reg_radix_ok(REG_THREE, 1, p1)) consider(true, p1, p2, p3, REG_THREE);
            }
        }
    }
    return best_cost >= 0;
}

int reg_threads(const RegFft &F, int count, int most) {
    long long best = -1;
    int threads = 64;
    for (int t = 64; t <= most; t += 64) {
        long long c = 0;
        for (int k = 0; k < F.nsteps; k++) {
            const long long rounds = ((long long)F.st[k].items * count + t - 1) / t;
            c += rounds * line_cost(F.st[k].radix);
        }
        if (best < 0 || c < best) {
            best = c;
            threads = t;
        }
    }
    return threads;
}

namespace {

using Z = std::complex<double>;

// exp(+2 pi i num / den)
Z unit(long long num, long long den) {
    const double a = 2.0 * M_PI * double(num % den) / double(den);
    return Z(std::cos(a), std::sin(a));
}

// Transform of length m, sign +1, in double: out[k] = sum_t in[t stride] w[t k * (M / m)], by the smallest
// prime factor; w holds the M-th roots of unity.
void host_dft(const Z *in, Z *out, int m, int stride, const std::vector<Z> &w) {
    const int M = int(w.size());
    if (m == 1) {
        out[0] = in[0];
        return;
    }
    int p = 2;
    while (m % p) p++;
    const int q = m / p;
    std::vector<Z> sub(m);
    for (int r = 0; r < p; r++) host_dft(in + r * stride, sub.data() + r * q, q, stride * p, w);
    for (int k = 0; k < m; k++) {
        Z acc = 0.0;
        for (int r = 0; r < p; r++) acc += sub[r * q + k % q] * w[size_t((long long)r * k % m) * (M / m)];
        out[k] = acc;
    }
}

float2 f2(const Z &z) { return make_float2(float(z.real()), float(z.imag())); }

}  // namespace

void reg_tables(const RegFft &F, RegTables &t) {
    const int m = F.m, p1 = F.st[0].radix;
    const int p2 = F.st[1].radix, p3 = F.stages == 3 ? F.st[2].radix : 1;
    t.data.clear();
    // twiddle of point r of line i of step k
    auto fill = [&](auto value) {
        for (int e = 0; e < m; e++) t.data.push_back(f2(value(e)));
    };
    for (int k = 0; k < F.nsteps; k++) {
        const RegStep &S = F.st[k];
        if (S.tw < 0) continue;
        if (k == 0) {  // after axis 1: W_m^(k1 (n2 p3 + n3))
            fill([&](int e) { return unit((long long)(e / S.items) * (e % S.items), m); });
        } else if (F.stages == 2) {  // back from axis 2: line k1, point n2: W_m^(n2 k1)
            fill([&](int e) { return unit((long long)(e / S.items) * (e % S.items), m); });
        } else if (k == 1) {  // after axis 2: line (k1, n3), point k2: W_(p2 p3)^(k2 n3)
            fill([&](int e) { return unit((long long)(e / S.items) * ((e % S.items) % p3), p2 * p3); });
        } else if (k == 2) {  // back from axis 3: line (k1, k2) = k1 + p1 k2, point n3: W_(p2 p3)^(n3 k2)
            fill([&](int e) { return unit((long long)(e / S.items) * ((e % S.items) / p1), p2 * p3); });
        } else {  // back from axis 2: line (k1, n3) = k1 p3 + n3, point n2: W_m^((n2 p3 + n3) k1)
            fill([&](int e) {
                const int i = e % S.items, n2 = e / S.items;
                return unit((long long)(n2 * p3 + i % p3) * (i / p3), m);
            });
        }
    }
    if (!F.blue) return;
    const int n = F.n;
    std::vector<Z> c(n), b(m, Z(0.0)), bt(m), w(m);
    for (int i = 0; i < n; i++) {
        const double a = M_PI * double((long long)i * i % (2LL * n)) / double(n);
        c[i] = Z(std::cos(a), std::sin(a));
    }
    for (int d = 0; d < n; d++) {
        b[d] = std::conj(c[d]);
        if (d) b[m - d] = std::conj(c[d]);
    }
    for (int i = 0; i < m; i++) w[i] = unit(i, m);
    host_dft(b.data(), bt.data(), m, 1, w);
    t.chirp = t.data.size();
    for (int i = 0; i < n; i++) t.data.push_back(f2(c[i]));
    t.bhat = t.data.size();
    for (int i = 0; i < m; i++) t.data.push_back(f2(bt[i] / double(m)));
}

const RegFft *reg_fft_len(iqm_ctx *ctx, int n, int &kind) {
    auto it = ctx->reg_plans.find(n);
    if (it == ctx->reg_plans.end()) {
        auto plan = std::make_unique<RegPlan>();
        if (reg_plan(n, plan->fft, plan->kind)) {
            RegTables t;
            reg_tables(plan->fft, t);
            const size_t bytes = sizeof(float2) * t.data.size();
            if (cudaMalloc(&plan->dev, bytes) != cudaSuccess) {
                cudaGetLastError();
                throw Error{IQM_ENOMEM, "FFT table allocation failed"};
            }
            IQM_CHECK_CUDA(cudaMemcpy(plan->dev, t.data.data(), bytes, cudaMemcpyHostToDevice));
            const auto *p = static_cast<const float2 *>(plan->dev);
            plan->fft.tw = p;
            plan->fft.chirp = p + t.chirp;
            plan->fft.bhat = p + t.bhat;
        }
        it = ctx->reg_plans.emplace(n, plan.get()).first;
        plan.release();
    }
    kind = it->second->kind;
    return kind >= 0 ? &it->second->fft : nullptr;
}

}  // namespace iqm

void iqm_release_reg_plans(iqm_ctx *ctx) {
    for (auto &kv : ctx->reg_plans) delete kv.second;
    ctx->reg_plans.clear();
}
