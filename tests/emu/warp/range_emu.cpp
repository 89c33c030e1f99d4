// Runs fix_range_kernel and fix_keeps_fp64 (stablercwa_gb300/csrc/eig_fixed.cuh) on the CPU: which matrices the fixed-point eigensolvers leave to
// the FP64 kernels, whose small eigenvalues those keep relative to themselves, and which they take (layer matrices of every
// declared kind among them).
#include <random>

#include "fibers.h"

#include "../../../stablercwa_gb300/csrc/eig_fixed.cuh"

using namespace rcwa_gb300;
static int failures = 0;
using M = std::vector<zc>;

template <bool Herm>
static void check(const char* name, int n, const M& a, bool other) {
    for (bool descending : {false, true}) {
        if (descending && n > 2) break;
        int status = -1;
        int flags[48] = {};
        if (Herm) run_cta(kFixRangeThreads, fix_range_smem(n), [&] { fix_range_kernel(n, 1, a.data(), (long long)n * n, &status, 2); }, descending);
        else run_cta(128, 0, [&] {
            const bool keep = fix_keeps_fp64(n, a.data(), flags);
            if (threadIdx.x == 77) status = keep ? 2 : 0;
        }, descending);
        const bool ok = status == (other ? 2 : 0);
        std::printf("%s %-36s n=%3d %s: %s\n", ok ? "pass" : "FAIL", name, n, Herm ? "Hermitian" : "general", status ? "FP64" : "fixed point");
        failures += !ok;
    }
}

static std::mt19937_64 rng(3);
static M random(int n, bool herm) {
    std::normal_distribution<double> g;
    M a((size_t)n * n);
    for (int j = 0; j < n; ++j)
        for (int i = 0; i < n; ++i) a[(size_t)j * n + i] = zc{g(rng), g(rng)};
    if (herm)
        for (int j = 0; j < n; ++j)
            for (int i = 0; i <= j; ++i) {
                if (i == j) a[(size_t)j * n + i].im = 0;
                a[(size_t)i * n + j] = conj(a[(size_t)j * n + i]);
            }
    return a;
}
// entries times f(i) g(j)
template <class F, class G>
static M scaled(int n, M a, F f, G g) {
    for (int j = 0; j < n; ++j)
        for (int i = 0; i < n; ++i) a[(size_t)j * n + i] = a[(size_t)j * n + i] * (f(i) * g(j));
    return a;
}
static M diagonal(int n, double (*f)(int, int)) {
    M a((size_t)n * n, zc{0, 0});
    for (int i = 0; i < n; ++i) a[(size_t)i * n + i] = zc{f(i, n), 0};
    return a;
}
// Kx^2 - [[eps]] of a two-segment profile: orders sin(theta) - m lambda / period
static M layer(int n, double step, double s, double e1, double e2, double loss, double fill) {
    const double pi = std::acos(-1.0);
    M a((size_t)n * n);
    for (int j = 0; j < n; ++j)
        for (int i = 0; i < n; ++i) {
            const int h = i - j;
            const double c = h ? std::sin(pi * h * fill) / (pi * h) : fill;
            zc v{-(e1 - e2) * c - (h ? 0.0 : e2), -loss * c};
            if (!h) {
                const double k = s - (i - n / 2) * step;
                v.re += k * k;
            }
            a[(size_t)j * n + i] = v;
        }
    return a;
}

int main() {
    const auto one = [](int) { return 1.0; };
    for (int n : {2, 30, 65}) {
        const auto down = [&](int i) { return std::pow(10.0, -5.0 * i / (n - 1)); };
        const auto down3 = [&](int i) { return std::pow(10.0, -3.0 * i / (n - 1)); };
        const auto up = [&](int i) { return std::pow(10.0, -5.0 * (n - 1 - i) / (n - 1)); };
        const M g = random(n, false), h = random(n, true);
        check<false>("random", n, g, false);
        check<true>("random", n, h, false);
        check<false>("random, 1e-250", n, scaled(n, g, [](int) { return 1e-250; }, one), false);
        check<false>("graded downwards over 1e-10", n, scaled(n, g, down, down), true);
        if (n > 2) check<true>("graded downwards over 1e-10", n, scaled(n, h, down, down), false);  // FP64 is no closer
        check<false>("graded downwards over 1e-6", n, scaled(n, g, down3, down3), true);
        check<false>("rows graded downwards", n, scaled(n, g, down, one), true);
        check<false>("columns graded downwards", n, scaled(n, g, one, down), true);
        if (n > 2) check<true>("graded upwards over 1e-10", n, scaled(n, h, up, up), false);
        M d = diagonal(n, [](int i, int n) { return std::pow(10.0, -20.0 * i / (n - 1)); });
        check<false>("diagonal, 1 to 1e-20", n, d, true);
        check<true>("diagonal, 1 to 1e-20", n, d, true);
        d[0] = zc{0, 0};
        if (n > 2) check<true>("diagonal, a zero row first", n, d, true);
        check<true>("diagonal, upwards", n, diagonal(n, [](int i, int n) { return std::pow(10.0, -20.0 * (n - 1 - i) / (n - 1)); }), true);
        check<true>("identity", n, diagonal(n, [](int, int) { return 1.0; }), false);
        check<true>("zero", n, M((size_t)n * n, zc{0, 0}), false);
        M u = g;
        for (int j = 0; j < n; ++j)
            for (int i = j + 1; i < n; ++i) u[(size_t)j * n + i] = zc{0, 0};
        check<false>("upper triangular", n, u, true);
        if (n < 24) continue;
        for (int lead : {2, n / 2, n - 1}) {  // rows `lead` on without entries left of the diagonal: deflated before any shift
            M st = u;
            for (int j = 0; j < lead; ++j)
                for (int i = 0; i < lead; ++i) st[(size_t)j * n + i] = g[(size_t)j * n + i];
            for (int i = 0; i < n; ++i) st[(size_t)i * n + i] = zc{1.0 + i, 0};
            check<false>("dense block, triangular rest", n, st, false);
            M one_small = st;
            one_small[(size_t)(n - 1 - (lead < n - 1)) * (n + 1)] = zc{1e-10, 0};
            check<false>("the same, a small diagonal entry", n, one_small, true);
            for (double small : {1e-20, 1e-5}) {
                M sm = st, sd = st;
                for (int j = 0; j < n; ++j)
                    for (int i = 0; i < n; ++i) {
                        const bool in = i < lead && j < lead;
                        sm[(size_t)j * n + i] = st[(size_t)j * n + i] * (in ? small : 1.0);
                        sd[(size_t)j * n + i] = st[(size_t)j * n + i] * (in ? small : i == j ? 1.0 : 0.0);
                    }
                check<false>("a small block first, triangular rest", n, sm, true);
                check<false>("a small block first, diagonal rest", n, sd, true);
            }
        }
        for (bool first : {false, true})  // two blocks of very different size, the small one first or last
            for (double small : {1e-20, 1e-5}) {
                M hb = h, gb = g;
                for (int j = 0; j < n; ++j)
                    for (int i = 0; i < n; ++i) {
                        const bool si = first ? i < n / 2 : i >= n / 2, sj = first ? j < n / 2 : j >= n / 2;
                        const double f = si != sj ? 0.0 : si ? small : 1.0;
                        hb[(size_t)j * n + i] = hb[(size_t)j * n + i] * f;
                        gb[(size_t)j * n + i] = gb[(size_t)j * n + i] * f;
                    }
                check<true>("two blocks", n, hb, true);
                check<false>("two blocks", n, gb, !first);  // the QR shifts pass over a first block
            }
        M t((size_t)n * n, zc{0, 0});
        for (int i = 0; i < n; ++i) {
            t[(size_t)i * n + i] = zc{up(i) * up(i), 0};
            if (i) t[(size_t)(i - 1) * n + i] = t[(size_t)i * n + i - 1] = zc{0.3 * up(i) * up(i - 1), 0};
        }
        check<true>("tridiagonal, upwards", n, t, true);
        M bad = g;
        bad[n + 3] = zc{INFINITY, 0};
        check<true>("not finite", n, bad, false);
    }
    for (int n : {25, 41, 121})
        for (double step : {0.1, 1.83, 10.0})
            for (double s : {0.01, 0.98}) {
                check<true>("lossless layer", n, layer(n, step, s, 2.13, 1.0, 0.0, 0.4), false);
                check<true>("lossless layer, high contrast", n, layer(n, step, s, 15.0, 1.0, 0.0, 0.6), false);
                check<true>("lossless layer, a few percent", n, layer(n, step, s, 2.13, 2.05, 0.0, 0.37), false);
                check<false>("absorbing layer", n, layer(n, step, s, 2.13, 1.0, 0.03, 0.5), false);
            }
    std::printf("%s\n", failures ? "FAILED" : "OK");
    return failures ? 1 : 0;
}
