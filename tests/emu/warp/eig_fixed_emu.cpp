// Runs the fixed-point eigensolver's kernels (stablercwa_gb300/csrc/eig_fixed.cuh) on the CPU through
// tests/emu/warp/cuda_runtime.h and checks, per case, against the matrix itself: ||Z^H Z - I||, the Schur
// residual ||Z^H A Z - T||_F / ||A||_F (the product in double), and the eigenpair residual ||A v - lambda v|| / (||A||_F ||v||).
// Bounds 1e-13 as for the FP64 solver. Exit status 0 and a final "OK" line when every case passes.
#include <complex>
#include <cstdio>
#include <functional>
#include <random>
#include <vector>

#include <ucontext.h>

#include "cuda_runtime.h"

dim3e threadIdx{0}, blockIdx{0}, blockDim{32};
unsigned char* emu_smem;
uint64_t emu_slot[1024];

namespace {
constexpr size_t kStack = 256 * 1024;
struct Fiber {
    ucontext_t ctx;
    std::vector<char> stack;
    int state = 0;  // 0 runs, 1 at a warp barrier, 2 at the CTA's, 3 done
};
std::vector<Fiber> fibers;
ucontext_t scheduler;
const std::function<void()>* body;
void entry() {
    (*body)();
    fibers[threadIdx.x].state = 3;
    swapcontext(&fibers[threadIdx.x].ctx, &scheduler);
}
void wait_at(int state) {
    const unsigned me = threadIdx.x;
    fibers[me].state = state;
    swapcontext(&fibers[me].ctx, &scheduler);
    threadIdx.x = me;
}
// one CTA of `threads` fibers running f, with `bytes` of dynamic shared memory
void run_cta(int threads, size_t bytes, const std::function<void()>& f) {
    std::vector<double> smem((bytes + 7) / 8);
    emu_smem = reinterpret_cast<unsigned char*>(smem.data());
    fibers.resize(threads);
    body = &f;
    blockDim.x = threads;
    for (int k = 0; k < threads; ++k) {
        Fiber& b = fibers[k];
        b.stack.resize(kStack);
        getcontext(&b.ctx);
        b.ctx.uc_stack.ss_sp = b.stack.data();
        b.ctx.uc_stack.ss_size = kStack;
        b.ctx.uc_link = nullptr;
        makecontext(&b.ctx, entry, 0);
        b.state = 0;
    }
    for (;;) {
        bool any = false;
        for (int k = 0; k < threads; ++k)
            if (fibers[k].state == 0) {
                any = true;
                threadIdx.x = k;
                swapcontext(&scheduler, &fibers[k].ctx);
            }
        int done = 0, at_block = 0;
        for (int w = 0; w < threads; w += 32) {
            int at = 0, gone = 0;
            for (int k = w; k < w + 32; ++k) {
                at += fibers[k].state == 1;
                gone += fibers[k].state == 3;
                at_block += fibers[k].state == 2;
            }
            done += gone;
            if (at && at + gone == 32)
                for (int k = w; k < w + 32; ++k)
                    if (fibers[k].state == 1) fibers[k].state = 0, any = true;
        }
        if (done == threads) return;
        if (at_block && at_block + done == threads)
            for (int k = 0; k < threads; ++k)
                if (fibers[k].state == 2) fibers[k].state = 0, any = true;
        if (!any) {
            std::printf("FAIL: the emulated threads wait for one another\n");
            std::exit(1);
        }
    }
}
}  // namespace
void emu_block_sync() { wait_at(2); }
void emu_warp_sync() { wait_at(1); }

#include "../../../stablercwa_gb300/csrc/eig_fixed.cuh"

using namespace rcwa_gb300;
using cd = std::complex<double>;
using M = std::vector<zc>;
static int failures = 0;

static M product(int n, const M& a, const M& b) {
    M c((size_t)n * n, zc{0, 0});
    for (int j = 0; j < n; ++j)
        for (int k = 0; k < n; ++k)
            for (int i = 0; i < n; ++i) c[(size_t)j * n + i] = zmac(a[(size_t)k * n + i], b[(size_t)j * n + k], c[(size_t)j * n + i]);
    return c;
}

static void solve(const char* name, int n, const M& a, int warps, int want_status) {
    const long long nn = (long long)n * n;
    std::vector<lz> H(nn);
    std::vector<int4> log(2 * fix_log_capacity(n)), table(fix_table_capacity(n));
    std::vector<zc> w(n), Z(nn);
    int head[2] = {0, 0}, status = -1, done = -1, info = -1;
    run_cta(32 * warps, fix_schur_smem(n, warps), [&] {
        fix_schur_kernel<false>(n, 1, a.data(), nn, w.data(), H.data(), nn, log.data(), (long long)log.size(), table.data(), head, &status, &done, &info);
    });
    if (status != want_status || done != !status) {
        std::printf("FAIL %s n=%d: status %d done %d\n", name, n, status, done);
        ++failures;
        return;
    }
    if (status) {
        std::printf("pass %-22s n=%3d left to the FP64 kernels\n", name, n);
        return;
    }
    for (int by = 0; by * 32 < n; ++by) {
        blockIdx.y = by;
        run_cta(32, (size_t)n * 32 * sizeof(lz), [&] { fix_apply_kernel(n, 1, Z.data(), nn, log.data(), (long long)log.size(), table.data(), head, &status); });
    }
    blockIdx.y = 0;
    M Zh(nn);
    for (int j = 0; j < n; ++j)
        for (int i = 0; i < n; ++i) Zh[(size_t)j * n + i] = conj(Z[(size_t)i * n + j]);
    double fro = 0, orth = 0, schur = 0, worst = 0;
    for (const zc& z : a) fro += norm2(z);
    fro = std::sqrt(fro);
    const M eye = product(n, Zh, Z);
    for (int j = 0; j < n; ++j)
        for (int i = 0; i < n; ++i) orth = std::max(orth, zabs(eye[(size_t)j * n + i] - zc{i == j ? 1.0 : 0.0, 0.0}));
    M T(nn);
    unsigned long long tn = 0;
    blockDim.x = 1;
    for (long long k = 0; k < nn; ++k) {
        blockIdx.x = (unsigned)k;
        threadIdx.x = 0;
        fix_triangle_kernel(n, 1, H.data(), nn, T.data(), nn, w.data(), head, &status, &tn);
    }
    blockIdx.x = 0;
    const M exactT = product(n, Zh, product(n, a, Z));
    for (long long k = 0; k < nn; ++k) schur += norm2(exactT[k] - T[k]);
    schur = std::sqrt(schur) / fro;
    M X(nn);
    for (int by = 0; by * 32 < n; ++by) {
        blockIdx.y = by;
        run_cta(kFixBackThreads, (size_t)(n + 4) * 32 * sizeof(zc), [&] { fix_backsub_kernel(n, 1, T.data(), nn, w.data(), &tn, X.data(), nn, &status, 2.220446049250313e-16); });
    }
    blockIdx.y = 0;
    const M V = product(n, Z, X), AV = product(n, a, V);
    for (int j = 0; j < n; ++j) {
        double r = 0, v = 0;
        for (int i = 0; i < n; ++i) {
            r += norm2(AV[(size_t)j * n + i] - w[j] * V[(size_t)j * n + i]);
            v += norm2(V[(size_t)j * n + i]);
        }
        worst = std::max(worst, std::sqrt(r / v) / fro);
    }
    long long rot = 0;
    for (int k = 0; k < head[0]; ++k) rot += table[k].y - table[k].x;
    const bool ok = orth <= 1e-13 && schur <= 1e-13 && worst <= 1e-13;
    std::printf("%s %-22s n=%3d warps %d: sweeps %d rotations %.2f n^2, orthogonality %.1e, Schur residual %.1e, eigenpairs %.1e\n",
                ok ? "pass" : "FAIL", name, n, warps, head[0], (double)rot / nn, orth, schur, worst);
    failures += !ok;
}

// The Hermitian solver's pieces: the reduction to tridiagonal form, Q from its log, the QL kernel, its rotations on a
// real identity (herm_apply_real_kernel), V = Q Y.
static void solve_hermitian(const char* name, int n, const M& a, int warps, int want_left) {
    const long long nn = (long long)n * n;
    std::vector<zc> ws(eig_workspace_elems(n)), w(n), Q(nn);
    std::vector<int4> log(2 * fix_reduce_capacity(n)), table(1);
    std::vector<double> Y(nn);
    int head[2] = {0, 0}, status = -1, info = -1;
    unsigned long long rot = 0;
    run_cta(32 * warps, fix_schur_smem(n, warps), [&] {
        fix_schur_kernel<true>(n, 1, a.data(), nn, w.data(), reinterpret_cast<lz*>(ws.data()), 0, log.data(), (long long)log.size(), table.data(), head,
                               &status, nullptr, nullptr);
    });
    run_cta(32, (size_t)2 * n * kHermQlThreads * 8, [&] { herm_ql_fixed_kernel(n, 1, w.data(), &info, ws.data(), &status, &rot); });
    const int left = reinterpret_cast<const int*>(ws.data() + 3 * nn)[1];
    if (left != want_left || info != 0) {
        std::printf("FAIL %s n=%d: left %d info %d\n", name, n, left, info);
        ++failures;
        return;
    }
    if (left) {
        std::printf("pass %-22s n=%3d Hermitian, left to the FP64 kernels\n", name, n);
        return;
    }
    for (int by = 0; by * 32 < n; ++by) {
        blockIdx.y = by;
        run_cta(32, (size_t)n * 32 * sizeof(lz), [&] { fix_apply_kernel(n, 1, Q.data(), nn, log.data(), (long long)log.size(), table.data(), head, &status); });
        run_cta(32, (size_t)n * 32 * 8, [&] { herm_apply_real_kernel(n, 1, Y.data(), ws.data(), &info); });
    }
    blockIdx.y = 0;
    M Yc(nn), h(nn);
    for (long long k = 0; k < nn; ++k) Yc[k] = zc{Y[k], 0};
    for (int j = 0; j < n; ++j)
        for (int i = 0; i < n; ++i) {
            const zc x = a[(size_t)j * n + i], y = a[(size_t)i * n + j];
            h[(size_t)j * n + i] = zc{0.5 * (x.re + y.re), 0.5 * (x.im - y.im)};
        }
    const M V = product(n, Q, Yc), HV = product(n, h, V);
    double fro = 0, orth = 0, worst = 0;
    for (const zc& z : h) fro += norm2(z);
    fro = std::sqrt(fro);
    for (int j = 0; j < n; ++j) {
        double r = 0;
        for (int i = 0; i < n; ++i) r += norm2(HV[(size_t)j * n + i] - w[j].re * V[(size_t)j * n + i]);
        worst = std::max(worst, std::sqrt(r) / fro);
        for (int k = 0; k <= j; ++k) {
            zc s{0, 0};
            for (int i = 0; i < n; ++i) s = zmacc(V[(size_t)k * n + i], V[(size_t)j * n + i], s);
            orth = std::max(orth, zabs(s - zc{j == k ? 1.0 : 0.0, 0}));
        }
    }
    const bool ok = orth <= 1e-13 && worst <= 1e-13;
    std::printf("%s %-22s n=%3d Hermitian: rotations %.2f n^2, orthogonality %.1e, eigenpairs %.1e\n", ok ? "pass" : "FAIL", name, n,
                (double)rot / nn, orth, worst);
    failures += !ok;
}

int main() {
    std::mt19937_64 rng(7);
    std::normal_distribution<double> g;
    const auto random = [&](int n, double scale) {
        M a((size_t)n * n);
        for (zc& z : a) z = zc{scale * g(rng), scale * g(rng)};
        return a;
    };
    // an absorbing grating's TE matrix Kx^2 - [[eps]]
    const auto layer = [&](int n, double loss) {
        M a((size_t)n * n);
        const double f = 0.4, k = 1.05 / 0.574;
        for (int j = 0; j < n; ++j)
            for (int i = 0; i < n; ++i) {
                const int h = i - j;
                const cd c1 = h ? cd(0, 1) * (std::polar(1.0, -2 * M_PI * h * f) - 1.0) / (2 * M_PI * h) : cd(f);
                const cd eps = (h ? cd(0) : cd(1)) + (cd(2.1316, loss) - 1.0) * c1;
                const double kx = 0.87 - (j - n / 2) * k;
                a[(size_t)j * n + i] = zc{(h ? 0 : kx * kx) - eps.real(), -eps.imag()};
            }
        return a;
    };
    // rotations: q, s against long double
    {
        double worst = 0, unit = 0;
        std::uniform_real_distribution<double> u(-1, 1);
        for (int k = 0; k < 200000; ++k) {
            const int sa = rng() % 60, sb = rng() % 60, sc = rng() % 60;
            long long x = (long long)(u(rng) * 0x1p61) >> sa, y = (long long)(u(rng) * 0x1p61) >> sb, s = (long long)(u(rng) * 0x1p61) >> sc;
            if (k % 7 == 0) x = 0;
            if (k % 11 == 0) y = 0;
            if (k % 13 == 0) s = k % 2 ? 1 : -((1LL << 61) - 1);
            if (!(x | y | s)) continue;
            const FixRot r = fix_rotation(x, y, s);
            const long double nrm = std::sqrt((long double)x * x + (long double)y * y + (long double)s * s);
            const auto val = [](int h, int l) { return (((long double)h) * 0x1p30L + l) * 0x1p-60L; };
            const long double c = val(r.cr1, r.cr0), d = val(r.ci1, r.ci0), e = val(r.s1, r.s0);
            worst = std::max(worst, (double)std::max({std::fabs(c - x / nrm), std::fabs(d - y / nrm), std::fabs(e - s / nrm)}));
            unit = std::max(unit, (double)std::fabs(c * c + d * d + e * e - 1.0L));
        }
        const bool ok = worst <= 8 * 0x1p-60 && unit <= 16 * 0x1p-60;
        std::printf("%s rotations: coefficients off by %.2f units of 2^-60, |q|^2 + s^2 - 1 by %.2f\n", ok ? "pass" : "FAIL",
                    worst * 0x1p60, unit * 0x1p60);
        failures += !ok;
    }
    for (int n : {2, 3, 5, 17, 31, 32, 33, 34, 48, 64, 65, 66, 97}) solve("random", n, random(n, 1.0), n % 2 ? 4 : 2, 0);
    solve("random, small scale", 40, random(40, 1e-30), 4, 0);
    solve("random, large scale", 40, random(40, 1e40), 4, 0);
    for (int n : {25, 41, 121}) solve("absorbing grating", n, layer(n, 0.03), 4, 0);
    solve("lossless grating", 61, layer(61, 0.0), 3, 0);
    solve("wide", 161, layer(161, 0.2), 6, 0);
    {
        M a((size_t)50 * 50, zc{0, 0});  // diagonal, repeated entries
        for (int i = 0; i < 50; ++i) a[(size_t)i * 50 + i] = zc{(double)(i / 5), 1.0};
        solve("diagonal, repeated", 50, a, 4, 0);
        for (int i = 0; i + 1 < 50; ++i) a[(size_t)(i + 1) * 50 + i] = zc{0.5, 0.0};  // upper triangular
        solve("triangular, repeated", 50, a, 4, 0);
        M b((size_t)36 * 36, zc{0, 0});  // cyclic shift: eigenvalues on the unit circle, zero diagonal
        for (int i = 0; i < 36; ++i) b[(size_t)i * 36 + (i + 1) % 36] = zc{1.0, 0.0};
        solve("cyclic shift", 36, b, 4, 1);  // needs an exceptional shift
        M c = random(40, 1.0);  // two blocks of very different size
        for (int j = 0; j < 40; ++j)
            for (int i = 0; i < 40; ++i) {
                if ((i < 20) != (j < 20)) c[(size_t)j * 40 + i] = zc{0, 0};
                else if (i >= 20) c[(size_t)j * 40 + i] = c[(size_t)j * 40 + i] * 1e-6;
            }
        solve("two scales", 40, c, 4, 0);
        solve("zero", 30, M((size_t)900, zc{0, 0}), 4, 1);
        M d = random(30, 1.0);
        d[77].im = NAN;
        solve("not finite", 30, d, 4, 1);
        solve("tiny", 30, random(30, 1e-290), 4, 1);
    }
    for (int n : {2, 3, 17, 32, 33, 65, 97}) solve_hermitian("random", n, random(n, 1.0), 4, 0);
    solve_hermitian("random, small scale", 40, random(40, 1e-30), 4, 0);
    for (int n : {41, 121}) solve_hermitian("lossless grating", n, layer(n, 0.0), 4, 0);
    {
        M a((size_t)50 * 50, zc{0, 0}), w21((size_t)41 * 41, zc{0, 0});
        for (int i = 0; i < 50; ++i) a[(size_t)i * 50 + i] = zc{(double)(i / 5) - 3, 0.0};
        solve_hermitian("diagonal, repeated", 50, a, 4, 0);
        for (int i = 0; i < 41; ++i) {  // Wilkinson's W+: pairs of eigenvalues equal to many digits
            w21[(size_t)i * 41 + i] = zc{std::fabs(i - 20.0), 0};
            if (i) w21[(size_t)i * 41 + i - 1] = w21[(size_t)(i - 1) * 41 + i] = zc{1, 0};
        }
        solve_hermitian("Wilkinson W+", 41, w21, 4, 0);
        solve_hermitian("zero", 30, M((size_t)900, zc{0, 0}), 4, 1);
    }
    std::printf("%s\n", failures ? "FAILED" : "OK");
    return failures ? 1 : 0;
}
