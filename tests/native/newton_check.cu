// Accuracy check of the refined square root and reciprocal of M-SVD's singular values and of FSIM's square root
// (iqm_internal.cuh): each runs on the GPU over seeded inputs, beside CUDA's own function, and the host
// prints "<name> <largest relative error> <the same of CUDA's function>" against double precision.
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <vector>

#include "iqm_internal.cuh"

namespace {

__global__ void eval(int kind, const float *x, int n, float *ours, float *cuda) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float a = x[i];
    switch (kind) {
        case 0: ours[i] = iqm::sqrt_newton(a); cuda[i] = sqrtf(a); break;
        case 1: ours[i] = iqm::rcp_newton(a); cuda[i] = 1.0f / a; break;
        default: ours[i] = iqm::sqrt_approx(a); cuda[i] = sqrtf(a); break;
    }
}

int check(int kind, const char *name, double lo, double hi, bool zero) {
    const int n = 1 << 21;
    std::vector<float> x(n), ours(n), cuda(n);
    uint64_t s = 977 + kind;
    for (int i = 0; i < n; i++) {
        s = s * 6364136223846793005ULL + 1442695040888963407ULL;
        const double u = double(s >> 11) * (1.0 / 9007199254740992.0);
        x[i] = float(lo * std::exp(u * std::log(hi / lo)));
    }
    if (zero) x[0] = 0.0f;
    float *d[3];
    for (auto &p : d)
        if (cudaMalloc(&p, n * sizeof(float))) return 1;
    cudaMemcpy(d[0], x.data(), n * sizeof(float), cudaMemcpyHostToDevice);
    eval<<<n / 256, 256>>>(kind, d[0], n, d[1], d[2]);
    if (cudaDeviceSynchronize() != cudaSuccess) return 1;
    cudaMemcpy(ours.data(), d[1], n * sizeof(float), cudaMemcpyDeviceToHost);
    cudaMemcpy(cuda.data(), d[2], n * sizeof(float), cudaMemcpyDeviceToHost);
    for (auto p : d) cudaFree(p);
    double worst = 0.0, worst_cuda = 0.0;
    for (int i = 0; i < n; i++) {
        const double ref = kind == 1 ? 1.0 / double(x[i]) : std::sqrt(double(x[i]));
        if (ref == 0.0) {
            if (ours[i] != 0.0f) worst = 1.0;
            continue;
        }
        worst = std::fmax(worst, std::fabs(ours[i] - ref) / ref);
        worst_cuda = std::fmax(worst_cuda, std::fabs(cuda[i] - ref) / ref);
    }
    std::printf("%s %.4e %.4e\n", name, worst, worst_cuda);
    return 0;
}

}  // namespace

int main() {
    // squared norms and singular values of 8x8 blocks, down to the smallest that are not taken as 0
    if (check(0, "sqrt_newton", 1e-30, 1e7, false)) return 1;
    // |x0| |x| + |x|^2 of a reflection
    if (check(1, "rcp_newton", 1e-30, 1e8, false)) return 1;
    // squared magnitudes of filter responses, and 0
    return check(2, "sqrt_approx", 1e-30, 1e20, true);
}
