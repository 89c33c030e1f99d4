// Runs the batched solvers' launchers on the host with the CUDA runtime's allocator and launches replaced (the linker's
// --wrap), lets the k-th allocation fail for every k, and checks that what was allocated before is given back. Nothing
// reaches a device: launches and copies do nothing.
#include <cstdio>
#include <functional>
#include <set>

#include "../../../stablercwa_gb300/csrc/engine.h"

using namespace rcwa_gb300;

static std::set<void*> live;
static long long calls, fail_at, next_address = 1 << 20;

extern "C" {
cudaError_t __wrap_cudaMallocAsync(void** p, size_t, cudaStream_t) {
    if (++calls == fail_at) return cudaErrorMemoryAllocation;
    *p = reinterpret_cast<void*>(next_address += 1 << 20);
    live.insert(*p);
    return cudaSuccess;
}
cudaError_t __wrap_cudaFreeAsync(void* p, cudaStream_t) {
    if (!live.erase(p)) std::printf("FAIL: freed what is not allocated\n");
    return cudaSuccess;
}
cudaError_t __wrap_cudaLaunchKernel(const void*, dim3, dim3, void**, size_t, cudaStream_t) { return cudaSuccess; }
cudaError_t __wrap_cudaGetLastError() { return cudaSuccess; }
cudaError_t __wrap_cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t __wrap_cudaGetDevice(int* d) { return *d = 0, cudaSuccess; }
cudaError_t __wrap_cudaMalloc(void** p, size_t) { return *p = reinterpret_cast<void*>(4096), cudaSuccess; }
cudaError_t __wrap_cudaMemset(void*, int, size_t) { return cudaSuccess; }
cudaError_t __wrap_cudaMemsetAsync(void*, int, size_t, cudaStream_t) { return cudaSuccess; }
cudaError_t __wrap_cudaMemcpy2DAsync(void*, size_t, const void*, size_t, size_t, size_t, cudaMemcpyKind, cudaStream_t) { return cudaSuccess; }
}

static int failures = 0;
static void check(const char* name, const std::function<void()>& launch) {
    int failed = 0;
    size_t kept = 0;
    for (fail_at = 1;; ++fail_at) {
        calls = 0;
        live.clear();
        try {
            launch();
        } catch (const EngineError&) {
            ++failed;
        }
        kept += live.size();
        if (calls < fail_at) break;  // all allocations succeeded
    }
    const bool ok = kept == 0 && failed >= 1;
    std::printf("%s %s: %lld allocations, %zu kept after a failure\n", ok ? "pass" : "FAIL", name, calls, kept);
    failures += !ok;
}

// allocations that only the fixed-point forms make: without one of them the FP64 kernels, which need less, take the call
static void answered(const char* name, const std::function<void()>& launch, int first, int last) {
    int refused = 0;
    size_t kept = 0;
    for (fail_at = first; fail_at <= last; ++fail_at) {
        calls = 0;
        live.clear();
        try {
            launch();
        } catch (const EngineError&) {
            ++refused;
        }
        kept += live.size();
    }
    const bool ok = refused == 0 && kept == 0;
    std::printf("%s %s: %d of %d calls refused, %zu kept\n", ok ? "pass" : "FAIL", name, refused, last - first + 1, kept);
    failures += !ok;
}

int main() {
    zc* d = reinterpret_cast<zc*>(1 << 16);
    int* info = reinterpret_cast<int*>(1 << 12);
    const double eps = 2.220446049250313e-16;
    const auto eig = [&](int n, int batch, zc* t) {
        return [=] { launch_eig(nullptr, n, batch, d, (long long)n * n, d, d, info, nullptr, d, eps, 30, 0, nullptr, 0, t); };
    };
    const auto herm = [&](int n, int batch) {
        return [=] { launch_eig_herm(nullptr, n, batch, d, (long long)n * n, d, d, info, d, eps, 30, 0); };
    };
    const auto lu = [&](int n, int nrhs, int batch) {
        return [=] {
            launch_lu_solve(nullptr, n, nrhs, batch, d, (long long)n * n, d, (long long)n * n, RHS_DENSE, d, (long long)n * nrhs, d,
                            (long long)n * nrhs, info);
        };
    };
    check("general eigensolver", eig(30, 3, nullptr));
    check("general eigensolver, its product on the tensor cores", eig(121, 500, nullptr));
    check("Schur form", eig(60, 3, d));
    check("Hermitian eigensolver, reduction by rotations", herm(41, 3));
    check("Hermitian eigensolver, lane groups", herm(20, 3));
    check("Hermitian eigensolver, panels", herm(121, 400));
    check("solve, warp panels", lu(41, 41, 700));
    check("solve, CTA panels", lu(121, 10, 2));
    check("solve with tensor-core updates", lu(121, 121, 100));
    check("product", [=] { launch_zgemm(nullptr, 64, 64, 80, 10, d, 64, 64 * 80, d, 80, 80 * 64, nullptr, 0, d, 64, 64 * 64, 1.0, 0.0); });
    // after `done`: the logs, their tables and flags, the product's digit planes
    answered("general eigensolver without the rotation logs", eig(30, 3, nullptr), 2, 6);
    answered("general eigensolver without the product's planes", eig(121, 500, nullptr), 2, 10);
    answered("Schur form without the rotation logs", eig(60, 3, d), 2, 6);
    // after Q, Y and the status: the log, its heads and flags
    answered("Hermitian eigensolver without the rotation log", herm(41, 3), 4, 6);
    std::printf("%s\n", failures ? "FAILED" : "OK");
    return failures ? 1 : 0;
}
