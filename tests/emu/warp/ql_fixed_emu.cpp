// Runs herm_ql_fixed_kernel (stablercwa_gb300/csrc/eig_fixed.cuh) on the CPU on the tridiagonal forms of lossless
// grating layers and compares every eigenvalue with bisection in long double. The eigenvalues that matter in a grating
// are small beside the matrix: no eigenvalue may be off by more than one FP64 rounding of an entry of the size of
// Gershgorin's bound N, 2^-54 N, however many rotations it took.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <vector>

#include "cuda_runtime.h"

dim3e threadIdx{0}, blockIdx{0}, blockDim{1};
unsigned char* emu_smem;
uint64_t emu_slot[1024];
// the QL kernel is one thread a matrix and meets no barrier
void emu_warp_sync() {}
void emu_block_sync() {}

#include "../../../stablercwa_gb300/csrc/eig_fixed.cuh"
using namespace rcwa_gb300;
typedef long double ld;

// d, e of the real symmetric n x n matrix a, by Householder reflections
static void tridiagonal(int n, std::vector<ld> a, std::vector<double>& d, std::vector<double>& e) {
    for (int k = 0; k + 1 < n; ++k) {
        std::vector<ld> v(n, 0), w(n, 0);
        ld s = 0, vw = 0;
        for (int i = k + 1; i < n; ++i) s += a[i * n + k] * a[i * n + k];
        const ld x = a[(k + 1) * n + k], beta = x >= 0 ? -std::sqrt(s) : std::sqrt(s);
        e[k] = (double)beta;
        for (int i = k + 1; i < n; ++i) v[i] = a[i * n + k];
        v[k + 1] -= beta;
        const ld h = s - x * beta;  // |v|^2 / 2
        if (h == 0) continue;
        for (int i = k + 1; i < n; ++i) {
            for (int j = k + 1; j < n; ++j) w[i] += a[i * n + j] * v[j];
            w[i] /= h;
            vw += v[i] * w[i];
        }
        for (int i = k + 1; i < n; ++i) w[i] -= vw / (2 * h) * v[i];
        for (int i = k + 1; i < n; ++i)
            for (int j = k + 1; j < n; ++j) a[i * n + j] -= v[i] * w[j] + w[i] * v[j];
        if (k + 2 == n) break;
    }
    for (int i = 0; i < n; ++i) d[i] = (double)a[i * n + i];
}

// the k-th smallest eigenvalue
static ld bisect(int n, const std::vector<double>& d, const std::vector<double>& e, int k, ld lo, ld hi) {
    for (int it = 0; it < 80; ++it) {
        const ld x = (lo + hi) / 2;
        int below = 0;
        ld q = 1;
        for (int i = 0; i < n; ++i) {
            q = d[i] - x - (i ? (ld)e[i - 1] * e[i - 1] / q : 0);
            if (q == 0) q = 1e-30L;
            below += q < 0;
        }
        (below > k ? hi : lo) = x;
    }
    return (lo + hi) / 2;
}

int main() {
    int failures = 0;
    const struct {
        int n;
        double index, fill;
    } cases[] = {{2, 3.5, 0.5}, {33, 1.46, 0.4}, {121, 1.46, 0.3}, {121, 3.8, 0.6}, {201, 3.5, 0.5}, {301, 3.9, 0.37}};
    for (const auto& c : cases) {
        const int n = c.n;
        std::vector<ld> a((size_t)n * n);
        for (int i = 0; i < n; ++i)
            for (int j = 0; j < n; ++j) {
                const int h = i - j;
                const ld kx = 0.87L - (j - n / 2) * 1.83L, contrast = (ld)c.index * c.index - 1;
                a[i * n + j] = h ? -contrast * std::sin(M_PIl * h * c.fill) / (M_PIl * h) : kx * kx - 1 - contrast * c.fill;
            }
        std::vector<double> d(n), e(n, 0.0);
        tridiagonal(n, a, d, e);
        ld N = 0;
        for (int i = 0; i < n; ++i) N = std::max(N, std::fabs((ld)d[i]) + std::fabs((ld)e[i]) + (i ? std::fabs((ld)e[i - 1]) : 0));
        std::vector<zc> ws(eig_workspace_elems(n)), w(n);
        double* src = reinterpret_cast<double*>(ws.data() + 2LL * n * n);
        for (int i = 0; i < n; ++i) {
            src[i] = d[i];
            src[n + i] = e[i];
        }
        std::vector<long long> smem((size_t)2 * n * kHermQlThreads);
        emu_smem = reinterpret_cast<unsigned char*>(smem.data());
        int info = -1, status = 0;
        unsigned long long rot = 0;
        herm_ql_fixed_kernel(n, 1, w.data(), &info, ws.data(), &status, &rot);
        const int left = reinterpret_cast<const int*>(ws.data() + 3LL * n * n)[1];
        std::vector<double> got(n);
        for (int i = 0; i < n; ++i) got[i] = w[i].re;
        std::sort(got.begin(), got.end());
        double worst = 0;
        for (int k = 0; k < n; ++k) {
            const ld x = bisect(n, d, e, k, -N, N), off = std::fabs(got[k] - x);
            // the eigenvalue's own rounding to FP64 is not the iteration's
            worst = std::max(worst, (double)((off - std::fabs(x) * 0x1p-53L) / N));
        }
        const bool ok = !left && info == 0 && worst <= 0x1p-54;
        std::printf("%s n=%3d index %.2f: worst eigenvalue off by %.2e N (2^%.1f), %.2f n^2 rotations\n", ok ? "pass" : "FAIL", n, c.index,
                    worst, std::log2(std::max(worst, 1e-30)), (double)rot / n / n);
        failures += !ok;
    }
    if (!failures) std::printf("OK\n");
    return failures != 0;
}
