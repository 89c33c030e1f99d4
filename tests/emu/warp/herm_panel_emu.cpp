// Runs the blocked Hermitian reduction's fixed-point panel (stablercwa_gb300/csrc/herm_fixed.cuh) on the CPU on matrices of
// one panel (order <= 33) and compares d and e with the FP64 panel's (eig.cuh herm_panel_one): both are backward stable,
// so they agree within 64 n eps N on dense matrices. Some matrices begin with columns that need no reflector. What the
// kernel leaves must depend neither on the order in which the lanes of a warp run between barriers nor on what an
// earlier user left in the workspace: bit for bit.
#include <random>

#include "fibers.h"

#include "../../../stablercwa_gb300/csrc/herm_fixed.cuh"

using namespace rcwa_gb300;
static int failures = 0;

struct Out {
    std::vector<double> de;
    std::vector<zc> v, m;
};

template <int G>
static Out run(int n, const std::vector<zc>& a, bool fixed, int stale, bool descending) {
    const long long nn = (long long)n * n;
    const int pnb = herm_panel_count(n) * kHermNb;
    std::vector<zc> ws(eig_workspace_elems(n)), pan(herm_panel_elems(n));
    int* w = reinterpret_cast<int*>(ws.data());
    for (size_t k = 0; k < ws.size() * 4; ++k) w[k] = stale;
    Out o{std::vector<double>(2 * n), std::vector<zc>(nn), std::vector<zc>((size_t)pnb * n)};
    run_cta(32, 0, [&] {
        if (fixed) herm_panel_fixed_kernel<G>(n, 1, 0, a.data(), nn, ws.data(), pan.data(), o.v.data(), o.m.data(), pnb);
        else if (threadIdx.x < G) herm_panel_one<G>(n, 0, a.data(), ws.data(), pan.data(), o.v.data(), o.m.data(), pnb);
    }, descending);
    std::memcpy(o.de.data(), ws.data() + 2 * nn, 2 * n * sizeof(double));
    return o;
}

template <int G>
static void check(const char* name, int n, const std::vector<zc>& a, bool dense) {
    double N = 0;
    for (int i = 0; i < n; ++i) {
        double s = 0;
        for (int j = 0; j < n; ++j) s += zabs(a[(size_t)j * n + i]);
        N = std::max(N, s);
    }
    const Out first = run<G>(n, a, true, 0, false), ref = run<G>(n, a, false, 0, false);
    double off = 0;
    for (int i = 0; i < 2 * n - 1; ++i) off = std::max(off, std::fabs(first.de[i] - ref.de[i]) / N);
    bool same = true;
    for (int stale : {0, -64, -65, -66, 0x40000000})
        for (bool descending : {false, true}) {
            const Out o = run<G>(n, a, true, stale, descending);
            same = same && std::memcmp(o.de.data(), first.de.data(), (2 * n - 1) * sizeof(double)) == 0 &&
                   std::memcmp(o.v.data(), first.v.data(), o.v.size() * sizeof(zc)) == 0 &&
                   std::memcmp(o.m.data(), first.m.data(), o.m.size() * sizeof(zc)) == 0;
        }
    const bool ok = same && (!dense || off <= 64 * n * 0x1p-52);
    std::printf("%s %-24s n=%2d G=%2d: d and e off FP64's by %.1e N, %s\n", ok ? "pass" : "FAIL", name, n, G, off,
                same ? "the same in every order" : "depends on the order or the workspace");
    failures += !ok;
}

int main() {
    std::mt19937_64 rng(5);
    std::normal_distribution<double> g;
    for (int n : {2, 3, 20, 32, 33}) {
        std::vector<zc> a((size_t)n * n);
        for (int j = 0; j < n; ++j)
            for (int i = 0; i <= j; ++i) {
                const zc v{g(rng), i == j ? 0.0 : g(rng)};
                a[(size_t)j * n + i] = v;
                a[(size_t)i * n + j] = conj(v);
            }
        check<4>("dense", n, a, true);
        check<32>("dense", n, a, true);
        for (int j = 0; j < n; ++j)
            for (int i = 0; i < n; ++i)
                if (std::min(i, j) < 4) {
                    a[(size_t)j * n + i] = zc{i == j ? 1.0 + i : std::abs(i - j) == 1 ? 0.5 : 0.0, 0.0};
                }
        check<4>("four columns reduced", n, a, true);
        check<8>("four columns reduced", n, a, true);
        check<32>("four columns reduced", n, a, true);
    }
    std::printf("%s\n", failures ? "FAILED" : "OK");
    return failures ? 1 : 0;
}
