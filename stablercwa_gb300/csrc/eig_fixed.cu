// eig_fixed.cu -- launcher of the fixed-point general eigensolver (kernels in eig_fixed.cuh).
#include <algorithm>
#include <cstdlib>

#include "herm_fixed.cuh"
#include "engine.h"

namespace rcwa_gb300 {
namespace {

// largest order: 32 rows of Z (16 bytes an entry) and the back substitution's slots in 227 KB of shared memory
constexpr int kFixMaxOrder = 440;
constexpr int kFixMinOrder = 24;
// Matrices per pass: the logs (about 96 n^2 bytes each) of half the batch, but of three matrices an SM at least and of
// 4 GB at most. The 2-D solver counts them in its estimate of a point; in the 1-D and conical ones they are freed before
// the dense operators that the estimate is made for come to be: calls with a limit of 1024 MiB held at most 942 (1-D,
// orders 31 to 301) and 987 MiB (conical, 25 to 121), absorbing or not, with one grating or three.
constexpr int kFixPassMin = 456;
constexpr long long kFixLogBytes = 4LL << 30;

// warps of fix_schur_kernel's CTA: a lane per row or column of the matrix up to order 352 (11 warps' tiles are
// what shared memory holds), at least four so that three warps trail the one that forms the rotations
int fix_warps(int n) { return std::min(11, std::max(4, (n + 31) / 32)); }

// Rows a CTA of the log's application: 32, or 16 where shared memory holds one CTA of 32 rows an SM (order 222 on) and
// they are more than the SMs: two CTAs of 16 take an SM in the time of one of 32 (a chain of latencies). 16 matrices of
// order 301, 160 CTAs of 32 rows on 152 SMs: the order-301
// scan 136.6 to 132.5 ms.
template <int R>
void fix_apply_rows(cudaStream_t st, int n, int batch, zc* z, long long z_stride, const int4* log, long long log_stride,
                    const int4* table, const int* head, const int* status) {
    const size_t smem = (size_t)n * R * sizeof(lz);
    if (smem > 45 * 1024) ensure_smem_optin(reinterpret_cast<const void*>(fix_apply_kernel<R>), (int)smem);
    fix_apply_kernel<R><<<dim3((unsigned)batch, (unsigned)((n + R - 1) / R)), R, smem, st>>>(n, batch, z, z_stride, log, log_stride, table,
                                                                                            head, status);
    RCWA_CUDA(cudaGetLastError());
}
void fix_apply(cudaStream_t st, int n, int batch, zc* z, long long z_stride, const int4* log, long long log_stride, const int4* table,
               const int* head, const int* status) {
    if (n >= 222 && (long long)batch * ((n + 31) / 32) > 152)
        fix_apply_rows<16>(st, n, batch, z, z_stride, log, log_stride, table, head, status);
    else
        fix_apply_rows<32>(st, n, batch, z, z_stride, log, log_stride, table, head, status);
}

void fix_range(cudaStream_t st, int n, int batch, const zc* a, long long a_stride, int* status, int other) {
    // Small CTAs where there are many matrices: they find room beside another stream's kernels (the mirror sweep, 4096 matrices
    // of order 121 a stream, 363.8 ms without this kernel: 365.1 with 64 threads, 365.8 with 128, 366.0 with 512).
    const int threads = batch >= 608 ? 64 : kFixRangeThreads;
    fix_range_kernel<<<(unsigned)batch, threads, fix_range_smem(n), st>>>(n, batch, a, a_stride, status, other);
    ++launch_count();
    RCWA_CUDA(cudaGetLastError());
}

}  // namespace

// RCWA_GB300_EIG_FIXED=0 keeps the FP64 iterations
bool eig_fixed_enabled() {
    static const bool on = [] {
        const char* e = std::getenv("RCWA_GB300_EIG_FIXED");
        return !(e && e[0] == '0');
    }();
    return on;
}

bool eig_fixed_possible(int n) { return eig_fixed_enabled() && n >= kFixMinOrder && n <= kFixMaxOrder; }

long long eig_fixed_bytes(int n) {
    if (!eig_fixed_possible(n)) return 0;
    return 2 * fix_log_capacity(n) * (long long)sizeof(int4) + fix_table_capacity(n) * (long long)sizeof(int4);
}

void launch_eig_fixed(cudaStream_t st, int n, int batch, const zc* a, long long a_stride, zc* w, zc* v, int* info, zc* ws,
                      int* done, double eps, zc* t_out) {
    const long long nn = (long long)n * n, wst = (3 * nn + 4LL * n + 8);  // eig_workspace_elems
    const int warps = fix_warps(n);
    const size_t schur_smem = fix_schur_smem(n, warps), back_smem = (size_t)(n + 4) * 32 * sizeof(zc);
    ensure_smem_optin(reinterpret_cast<const void*>(fix_schur_kernel<false>), (int)schur_smem);
    if (back_smem > 48 * 1024) ensure_smem_optin(reinterpret_cast<const void*>(fix_backsub_kernel), (int)back_smem);
    const int chunk = (int)std::max(1LL, std::min<long long>(std::min(batch, std::max(kFixPassMin, (batch + 1) / 2)),
                                                             kFixLogBytes / eig_fixed_bytes(n)));
    DeviceScratch mem(st);
    int4* log = mem.get<int4>((size_t)chunk * 2 * fix_log_capacity(n));
    int4* table = mem.get<int4>((size_t)chunk * fix_table_capacity(n));
    int *head = mem.get<int>((size_t)chunk * 2), *status = mem.get<int>(chunk);
    unsigned long long* tn = mem.get<unsigned long long>(chunk);
    for (int b0 = 0; b0 < batch; b0 += chunk) {
        const int cb = std::min(chunk, batch - b0);
        const zc* ac = a + (long long)b0 * a_stride;
        zc *wc = w + (long long)b0 * n, *vc = v + (long long)b0 * nn, *wsc = ws + (long long)b0 * wst;
        zc *z1 = wsc + nn, *z2 = wsc + 2 * nn;  // Z; X
        lz* h = reinterpret_cast<lz*>(wsc);
        fix_schur_kernel<false><<<(unsigned)cb, 32 * warps, schur_smem, st>>>(n, cb, ac, a_stride, wc, h, wst, log, 2 * fix_log_capacity(n), table, head, status,
                                                                       done + b0, info + b0, nullptr, true);
        RCWA_CUDA(cudaGetLastError());
        fix_apply(st, n, cb, z1, wst, log, 2 * fix_log_capacity(n), table, head, status);
        zc* t = t_out ? t_out + (long long)b0 * nn : vc;
        RCWA_CUDA(cudaMemsetAsync(tn, 0, (size_t)cb * sizeof(unsigned long long), st));
        fix_triangle_kernel<<<(unsigned)((nn * cb + 255) / 256), 256, 0, st>>>(n, cb, h, wst, t, nn, wc, head, status, tn);
        RCWA_CUDA(cudaGetLastError());
        launch_count() += 3;
        if (t_out) {  // the Schur form: T and Z
            RCWA_CUDA(cudaMemcpy2DAsync(vc, nn * sizeof(zc), z1, wst * sizeof(zc), nn * sizeof(zc), cb, cudaMemcpyDeviceToDevice, st));
            continue;
        }
        fix_backsub_kernel<<<dim3((unsigned)cb, (unsigned)((n + 31) / 32)), kFixBackThreads, back_smem, st>>>(
            n, cb, t, nn, wc, tn, z2, wst, status, eps);
        RCWA_CUDA(cudaGetLastError());
        launch_zgemm_untimed(st, n, n, n, cb, z1, n, wst, z2, n, wst, nullptr, 0, vc, n, nn, 1.0, 0.0, status, 1);
        fix_unit_columns_kernel<<<(unsigned)(((long long)cb * n * 32 + 127) / 128), 128, 0, st>>>(n, cb, vc, nn, status);
        RCWA_CUDA(cudaGetLastError());
        launch_count() += 2;
    }
}

// status[b] = kFixOther for a matrix that the FP64 reduction and QL iteration keep, else 0
void launch_herm_range(cudaStream_t st, int n, int batch, const zc* a, long long a_stride, int* status) {
    fix_range(st, n, batch, a, a_stride, status, kFixOther);
}

// The Hermitian solver's reduction: d and e into ws (where the QL kernel reads them) and Q (n x n, contiguous);
// status[b] = 1 for a matrix left to the fused FP64 kernel.
void launch_herm_reduce_fixed(cudaStream_t st, int n, int batch, const zc* a, long long a_stride, zc* q, zc* ws, int* status) {
    const long long nn = (long long)n * n, wst = 3 * nn + 4LL * n + 8, log_stride = 2 * fix_reduce_capacity(n);
    const int warps = fix_warps(n);
    const size_t schur_smem = fix_schur_smem(n, warps);
    ensure_smem_optin(reinterpret_cast<const void*>(fix_schur_kernel<true>), (int)schur_smem);
    DeviceScratch mem(st);
    int4* log = mem.get<int4>((size_t)batch * log_stride);
    int *head = mem.get<int>((size_t)batch * 2), *other = mem.get<int>(batch);
    fix_range(st, n, batch, a, a_stride, other, 1);
    fix_schur_kernel<true><<<(unsigned)batch, 32 * warps, schur_smem, st>>>(n, batch, a, a_stride, nullptr, reinterpret_cast<lz*>(ws), wst,
                                                                            log, log_stride, nullptr, head, status, nullptr, nullptr, other);
    RCWA_CUDA(cudaGetLastError());
    fix_apply(st, n, batch, q, nn, log, log_stride, nullptr, head, status);
    launch_count() += 2;
}

void launch_herm_ql_fixed(cudaStream_t st, int n, int batch, zc* w, int* info, zc* ws, const int* status) {
    // A matrix a lane, and no more lanes a warp than give each SM one warp: lanes of a warp run sweeps of different
    // lengths, and the chain of one waits for the branches of the others (16 matrices of order 301: 65 ms in one warp,
    // 50 in a warp each; the scan of them 152 to 137 ms). One warp a scheduler (608 in all) leaves the other polarisation's stream less room: the
    // mirror sweep, 4096 matrices a stream, 381 against 372 ms.
    int lanes = 1;
    while (lanes < kHermQlThreads && 152LL * lanes < batch) lanes *= 2;
    const size_t smem = (size_t)2 * n * lanes * sizeof(long long);
    if (smem > 48 * 1024) ensure_smem_optin(reinterpret_cast<const void*>(herm_ql_fixed_kernel), (int)smem);
    herm_ql_fixed_kernel<<<(unsigned)((batch + lanes - 1) / lanes), lanes, smem, st>>>(
        n, batch, w, info, ws, status, rotation_counter());
    RCWA_CUDA(cudaGetLastError());
}

namespace {
template <int G>
void panel_launch(cudaStream_t st, int n, int batch, int k0, const zc* a, long long a_stride, zc* ws, zc* pan, zc* vall, zc* mall,
                  int pnb, const int* other) {
    const unsigned blocks = (unsigned)(((long long)batch * G + 127) / 128);
    herm_panel_fixed_kernel<G><<<blocks, 128, 0, st>>>(n, batch, k0, a, a_stride, ws, pan, vall, mall, pnb, other);
}
}  // namespace

void launch_herm_panel_fixed(cudaStream_t st, int n, int batch, int k0, const zc* a, long long a_stride, zc* ws, zc* pan, zc* vall,
                             zc* mall, int pnb, int group, const int* other) {
    switch (group) {
        case 4: panel_launch<4>(st, n, batch, k0, a, a_stride, ws, pan, vall, mall, pnb, other); break;
        case 8: panel_launch<8>(st, n, batch, k0, a, a_stride, ws, pan, vall, mall, pnb, other); break;
        case 16: panel_launch<16>(st, n, batch, k0, a, a_stride, ws, pan, vall, mall, pnb, other); break;
        case 32: panel_launch<32>(st, n, batch, k0, a, a_stride, ws, pan, vall, mall, pnb, other); break;
        default: throw EngineError{RCWA_EINVAL, "eig: the blocked Hermitian reduction takes 4, 8, 16 or 32 lanes"};
    }
    ++launch_count();
    RCWA_CUDA(cudaGetLastError());
}

}  // namespace rcwa_gb300
