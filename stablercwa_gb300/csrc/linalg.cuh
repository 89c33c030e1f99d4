// linalg.cuh -- batched complex FP64 LU solve and GEMM for sm_103a.
//
// Both are bound by the FP64 pipe (about 2 lane-FMAs per clock per SM on GB300), not by memory: a
// complex multiply-add is 4 FP64 FMAs per 16-32 bytes touched, and GB300's HBM/L2 deliver far more
// bytes per FP64 operation than that. So the kernels spend nothing on elaborate tiling; they keep
// every lane busy with independent FP64 work and read operands coalesced (column-major, lanes along
// rows) or as warp broadcasts.
#pragma once

#include "common.cuh"

namespace rcwa_gb300 {

// Batched A X = B with partial pivoting, one warp per system (include/stablercwa/lu.hpp:268-396 and
// :233-266). Pivot: first entry of largest |z| (hypot) at or below the diagonal; multipliers
// a*(1/pivot) unless 1/pivot overflows; a zero pivot marks the system singular and the step is
// skipped, exactly as the reference continues past it before refusing to solve. The right-hand
// sides are eliminated together with the matrix (an augmented sweep performs the same per-element
// operations, in the same order, as factor-then-forward-substitute), then back-substituted.
//
// a      : batch n x n (column-major), read; factored into lu (may alias a when in_place)
// rhs    : RHS_DENSE: batch n x nrhs; RHS_DIAG: batch n-vectors (nrhs = n); RHS_IDENTITY: none
// x      : batch n x nrhs output
// skip   : optional per-system flag; a nonzero entry leaves that system untouched
// singular: per-system output flag (set to 1 on a zero pivot, never cleared)
__global__ void __launch_bounds__(128) lu_solve_kernel(int n, int nrhs, int batch, const zc* a, long long a_stride,
                                                       zc* lu, long long lu_stride, int rhs_kind, const zc* rhs,
                                                       long long rhs_stride, zc* x, long long x_stride,
                                                       int* __restrict__ singular,
                                                       const int* __restrict__ skip, int skip_value) {
    const long long sys = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (sys >= batch) return;
    if (skip && skip[sys] == skip_value) return;
    const int lane = threadIdx.x & 31;
    const zc* A = a + sys * a_stride;
    zc* L = lu + sys * lu_stride;
    zc* Xs = x + sys * x_stride;
    const long long nn = (long long)n * n;
    if (L != A)
        for (long long i = lane; i < nn; i += 32) L[i] = A[i];
    const long long xn = (long long)n * nrhs;
    if (rhs_kind == RHS_DENSE) {
        const zc* Bs = rhs + sys * rhs_stride;
        if (Bs != Xs)
            for (long long i = lane; i < xn; i += 32) Xs[i] = Bs[i];
    } else {
        const zc* d = rhs_kind == RHS_DIAG ? rhs + sys * rhs_stride : nullptr;
        for (long long i = lane; i < xn; i += 32) {
            const int c = (int)(i / n), r = (int)(i - (long long)c * n);
            Xs[i] = r == c ? (d ? d[r] : zc{1.0, 0.0}) : zc{0.0, 0.0};
        }
    }
    __syncwarp();
    int sing = 0;
    for (int k = 0; k < n; ++k) {
        zc* ck = L + (long long)k * n;
        // pivot search: first index of the largest |z| in rows k..n-1
        double best = -1.0;
        int bi = n;
        for (int i = k + lane; i < n; i += 32) {
            const double v = zabs(ck[i]);
            if (v > best) {
                best = v;
                bi = i;
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const double ov = __shfl_xor_sync(0xffffffffu, best, o);
            const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
            if (ov > best || (ov == best && oi < bi)) {
                best = ov;
                bi = oi;
            }
        }
        const int p = (best < 0.0 || bi >= n) ? k : bi;  // all-NaN column: keep the diagonal
        if (p != k) {
            for (int c = lane; c < n; c += 32) {
                zc* col = L + (long long)c * n;
                const zc t = col[k];
                col[k] = col[p];
                col[p] = t;
            }
            for (int c = lane; c < nrhs; c += 32) {
                zc* col = Xs + (long long)c * n;
                const zc t = col[k];
                col[k] = col[p];
                col[p] = t;
            }
        }
        __syncwarp();
        const zc piv = ck[k];
        if (is_zero(piv)) {
            sing = 1;
            for (int i = k + 1 + lane; i < n; i += 32) ck[i] = zc{0.0, 0.0};
            __syncwarp();
            continue;
        }
        const zc inv = zinv(piv);
        const bool inv_ok = zfinite(inv);
        // multipliers for the rows this lane owns (at most 8 register slots; rows beyond stay in memory)
        for (int i = k + 1 + lane; i < n; i += 32) ck[i] = inv_ok ? ck[i] * inv : zdiv(ck[i], piv);
        // trailing update of matrix columns and right-hand sides: col[i] -= l_i * col[k]
        for (int c = k + 1; c < n + nrhs; ++c) {
            zc* col = c < n ? L + (long long)c * n : Xs + (long long)(c - n) * n;
            const zc t = col[k];
            if (is_zero(t)) continue;
            for (int i = k + 1 + lane; i < n; i += 32) col[i] = zfms(ck[i], t, col[i]);
        }
        __syncwarp();
    }
    if (sing) {
        // the reference refuses to solve (std::runtime_error); the solution is reported as NaN
        const double nan = __longlong_as_double(0x7ff8000000000000LL);
        for (long long i = lane; i < xn; i += 32) Xs[i] = zc{nan, nan};
        if (lane == 0) singular[sys] = 1;
        return;
    }
    // back substitution U X = Y
    if (nrhs >= 16) {
        // lanes own right-hand-side columns
        for (int c = lane; c < nrhs; c += 32) {
            zc* xc = Xs + (long long)c * n;
            for (int k = n - 1; k >= 0; --k) {
                const zc* uk = L + (long long)k * n;
                const zc xk = zdiv(xc[k], uk[k]);
                xc[k] = xk;
                if (is_zero(xk)) continue;
                for (int i = 0; i < k; ++i) xc[i] = zfms(uk[i], xk, xc[i]);
            }
        }
    } else {
        // lanes own rows
        for (int c = 0; c < nrhs; ++c) {
            zc* xc = Xs + (long long)c * n;
            for (int k = n - 1; k >= 0; --k) {
                const zc* uk = L + (long long)k * n;
                const zc xk = zdiv(xc[k], uk[k]);
                __syncwarp();
                if (lane == (k & 31)) xc[k] = xk;
                if (!is_zero(xk))
                    for (int i = lane; i < k; i += 32) xc[i] = zfms(uk[i], xk, xc[i]);
                __syncwarp();
            }
        }
    }
}

// ---------------------------------------------------------------- blocked LU for large n
//
// The same partial-pivot elimination of [A | B] as lu_solve_kernel, reorganised for orders where a
// warp per system cannot keep the trailing matrix anywhere near the FP64 pipe: panels of nb columns
// are factored by one CTA or warp per system (pivot search, multipliers, rank-1 updates inside the
// panel), the remaining columns of A and the right-hand sides take the panel's row swaps, their panel
// rows are solved with the unit lower triangle (same subtraction order as the unblocked sweep), and
// the trailing matrix and right-hand sides are updated with a product. Back substitution runs block
// by block from the bottom: a triangular solve of the block rows, then a product for the rows above.

__device__ __forceinline__ zc* aug_col(zc* L, zc* X, int n, int c) {
    return c < n ? L + (long long)c * n : X + (long long)(c - n) * n;
}

// lu = a (if distinct), x = rhs (dense, identity or diagonal)
__global__ void lu_init_kernel(int n, int nrhs, int batch, const zc* a, long long a_stride, zc* lu, long long lu_stride,
                               int rhs_kind, const zc* rhs, long long rhs_stride, zc* x, long long x_stride,
                               const int* __restrict__ skip, int skip_value) {
    const long long per = (long long)n * (n + nrhs);
    const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= (long long)batch * per) return;
    const long long sys = idx / per;
    if (skip && skip[sys] == skip_value) return;
    const long long e = idx - sys * per;
    const long long nn = (long long)n * n;
    if (e < nn) {
        const zc* A = a + sys * a_stride;
        zc* L = lu + sys * lu_stride;
        if (L != A) L[e] = A[e];
        return;
    }
    const long long xe = e - nn;
    zc* Xs = x + sys * x_stride;
    if (rhs_kind == RHS_DENSE) {
        const zc* Bs = rhs + sys * rhs_stride;
        if (Bs != Xs) Xs[xe] = Bs[xe];
    } else {
        const int c = (int)(xe / n), r = (int)(xe - (long long)c * n);
        const zc* d = rhs_kind == RHS_DIAG ? rhs + sys * rhs_stride : nullptr;
        Xs[xe] = r == c ? (d ? d[r] : zc{1.0, 0.0}) : zc{0.0, 0.0};
    }
}

// 1 / z by one reciprocal of |z|^2 where that is in range
__device__ __forceinline__ zc pivot_inverse(zc z) {
    const double size = norm2(z);
    const int h = __double2hiint(size);  // exponents 2^-960 .. 2^960
    if (h < 0x03f00000 || h >= 0x7bf00000) return zinv(z);
    const double s = 1.0 / size;
    return zc{z.re * s, -z.im * s};
}

// 1 / z with a correction step, for the back substitution: a product with it is as close as a Smith division
__device__ __forceinline__ zc pivot_inverse_refined(zc z) {
    const zc a = pivot_inverse(z);
    const zc b = zmac(a, zfms(z, a, zc{1.0, 0.0}), a);
    return zfinite(b) ? b : a;
}

// Pivot search on integers (an FP64 comparison costs a warp 64 cycles): the key of a magnitude is the bits of |z|^2, or
// of |z| where squares leave the range, its upper half plus one so that zero, below every magnitude, is left for NaN.
struct PivotKey {
    unsigned hi, lo;
    int row;
};
__device__ __forceinline__ PivotKey pivot_key(double v, int row) {
    const unsigned h = (unsigned)__double2hiint(v) + 1u;
    return v != v ? PivotKey{0u, 0u, row} : PivotKey{h, (unsigned)__double2loint(v), row};
}
__device__ __forceinline__ bool pivot_in_range(PivotKey k) { return k.hi - 0x03f00001u < 0x7bf00001u - 0x03f00001u; }
// the larger key; rows are offered in ascending order, so the first of equals stays
__device__ __forceinline__ void pivot_offer(PivotKey& best, PivotKey k) {
    if (k.hi > best.hi || (k.hi == best.hi && (k.lo > best.lo || (k.lo == best.lo && k.row < best.row)))) best = k;
}
__device__ __forceinline__ PivotKey pivot_reduce(PivotKey k) {
    const unsigned hi = __reduce_max_sync(0xffffffffu, k.hi);
    const unsigned lo = __reduce_max_sync(0xffffffffu, k.hi == hi ? k.lo : 0u);
    const int row = __reduce_min_sync(0xffffffffu, k.hi == hi && k.lo == lo ? k.row : 0x7fffffff);
    return PivotKey{hi, lo, row};
}

// Factor columns k0 .. k0+nb-1 (rows k0 .. n-1), one 128-thread CTA per system, the panel in shared memory (Smem: 512
// bytes a row, n - k0 <= kPanelSmemRows) or in place. Row swaps stay inside the panel; what they do to the columns
// outside goes to swaps (kSwapInts a system, then n - k0 of scratch in place): the row that ends up in panel row i, and
// the (destination, source) pairs of the rows below the panel. dinv gets the pivots' reciprocals.
// Bound by the FP64 pipe, an instruction of which takes 64 cycles a warp whatever its lanes do, four warps at a time:
// so the pivot search compares integers, the multipliers share one reciprocal of |pivot|^2, and the four warps split
// rows, and up to 64 rows also columns (warp = row block + blocks x column group): each group forms the multipliers
// from raw, its copy of the unscaled column, and group 0, whose first column is the next pivot column, searches it
// while it is in registers. Two barriers a column. Four panels of one system of order 121: 500 us; with
// 256 threads, hypot, FP64 comparisons and five barriers 927.
constexpr int kPanelSmemRows = 440;
constexpr int kSwapInts = 96;
template <bool Smem>
__global__ void __launch_bounds__(128) lu_panel_kernel(int n, int batch, zc* lu, long long lu_stride, int k0, int nb,
                                                       int* __restrict__ swaps, int swap_stride, zc* __restrict__ dinv,
                                                       int* __restrict__ sing_local, const int* __restrict__ skip, int skip_value) {
    RCWA_DYN_SMEM(zc, panel_sm);
    const long long sys = blockIdx.x;
    if (sys >= batch) return;
    if (skip && skip[sys] == skip_value) return;
    __shared__ PivotKey s_key[4];
    __shared__ zc s_raw[2][64];
    __shared__ int s_piv[32];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    zc* L = lu + sys * lu_stride + (long long)k0 * n + k0;
    const int m = n - k0, w = min(nb, m);
    const long long ld = Smem ? m : n;
    zc* P = Smem ? panel_sm : L;
    int* out = swaps + sys * swap_stride;
    int* perm = Smem ? reinterpret_cast<int*>(panel_sm + (long long)m * 32) : out + kSwapInts;  // the original row of each row
    const int blocks = m <= 32 ? 1 : m <= 64 ? 2 : 4, groups = 4 / blocks;
    const int row0 = (warp & (blocks - 1)) * 32 + lane, group = warp / blocks;
    if (Smem)
        for (int c = 0; c < w; ++c)
            for (int r = tid; r < m; r += 128) P[c * ld + r] = L[(long long)c * n + r];
    for (int r = tid; r < m; r += 128) perm[r] = r;
    __syncthreads();
    if (group == 0) {
        PivotKey best{0u, 0u, 0x7fffffff};
        for (int r = row0; r < m; r += 32 * blocks) {
            const zc v = P[r];
            if (groups > 1) s_raw[0][r] = v;
            pivot_offer(best, pivot_key(norm2(v), r));
        }
        best = pivot_reduce(best);
        if (lane == 0) s_key[warp] = best;
    }
    for (int j = 0; j < w; ++j) {
        zc* col = P + j * ld;
        __syncthreads();
        PivotKey key = s_key[0];
        for (int b = 1; b < blocks; ++b) pivot_offer(key, s_key[b]);
        if (!pivot_in_range(key)) {
            // the largest square is subnormal, zero, infinite or not a number: by |z|
            PivotKey best{0u, 0u, 0x7fffffff};
            for (int r = row0; r < m; r += 32 * blocks)
                if (r >= j) pivot_offer(best, pivot_key(zabs(col[r]), r));
            best = pivot_reduce(best);
            __syncthreads();
            if (group == 0 && lane == 0) s_key[warp] = best;
            __syncthreads();
            key = s_key[0];
            for (int b = 1; b < blocks; ++b) pivot_offer(key, s_key[b]);
        }
        const int p = key.hi == 0u ? j : key.row;  // all-NaN column: keep the diagonal
        const bool zero = key.hi == 1u && key.lo == 0u;
        zc* raw = groups > 1 ? s_raw[j & 1] : col;
        const zc piv = raw[p];
        const zc inv = pivot_inverse(piv);
        const bool inv_ok = zfinite(inv);
        if (groups == 1) __syncthreads();  // raw is the column itself: read before it is swapped
        if (p != j) {
            if (tid < w) {
                const zc t = P[tid * ld + j];
                P[tid * ld + j] = P[tid * ld + p];
                P[tid * ld + p] = t;
            }
            if (tid == 64) {
                const int t = perm[j];
                perm[j] = perm[p];
                perm[p] = t;
            }
        }
        if (tid == 64) s_piv[j] = p;
        if (tid == 0 && zero) sing_local[sys] = 1;
        // the raw copy's row p now holds what was row j
        const zc raw_j = groups > 1 ? raw[j] : zc{0.0, 0.0};
        __syncthreads();
        PivotKey best{0u, 0u, 0x7fffffff};
        for (int r = row0; r < m; r += 32 * blocks) {
            if (r <= j) continue;
            const zc x = groups > 1 ? (r == p ? raw_j : raw[r]) : col[r];
            const zc l = zero ? zc{0.0, 0.0} : inv_ok ? x * inv : zdiv(x, piv);
            if (group == 0) col[r] = l;
            int c = j + 1 + group;
            if (group == 0 && c < w) {
                zc v = P[c * ld + r];
                if (!zero) v = zfms(l, P[c * ld + j], v);
                P[c * ld + r] = v;
                if (groups > 1) s_raw[(j + 1) & 1][r] = v;
                pivot_offer(best, pivot_key(norm2(v), r));
                c += groups;
            }
            if (zero) continue;
#pragma unroll 4
            for (; c < w; c += groups) P[c * ld + r] = zfms(l, P[c * ld + j], P[c * ld + r]);
        }
        if (group == 0) {
            best = pivot_reduce(best);
            if (lane == 0) s_key[warp] = best;
        }
    }
    __syncthreads();
    if (Smem)
        for (int c = 0; c < w; ++c)
            for (int r = tid; r < m; r += 128) L[(long long)c * n + r] = P[c * ld + r];
    if (tid >= 64 && tid < 64 + w) dinv[sys * n + k0 + tid - 64] = pivot_inverse_refined(P[(tid - 64) * (ld + 1)]);
    if (tid < 32) {
        out[tid] = k0 + (tid < w ? perm[tid] : 0);
        const bool below = tid < w && s_piv[tid] >= w;
        out[32 + tid] = below ? k0 + s_piv[tid] : -1;
        out[64 + tid] = below ? k0 + perm[s_piv[tid]] : -1;
    }
}

// The same panel factorisation with one warp per system (rows strided over the lanes, warp shuffles for
// the pivot search, no block barriers): the form for many systems of moderate order, where a CTA per
// system spends most of its time in barriers. Same pivot rule and the same arithmetic per element as
// lu_panel_kernel, so the factors are identical.
__global__ void __launch_bounds__(128) lu_panel_warp_kernel(int n, int nrhs, int batch, zc* lu, long long lu_stride, zc* x,
                                                            long long x_stride, int k0, int nb, zc* __restrict__ dinv,
                                                            int* __restrict__ sing_local,
                                                            const int* __restrict__ skip, int skip_value) {
    const long long sys = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (sys >= batch) return;
    if (skip && skip[sys] == skip_value) return;
    const int lane = threadIdx.x & 31;
    zc* L = lu + sys * lu_stride;
    zc* X = x + sys * x_stride;
    const int kend = min(k0 + nb, n);
    for (int j = k0; j < kend; ++j) {
        zc* col = L + (long long)j * n;
        PivotKey best{0u, 0u, 0x7fffffff};
        for (int i = j + lane; i < n; i += 32) pivot_offer(best, pivot_key(norm2(col[i]), i));
        best = pivot_reduce(best);
        if (!pivot_in_range(best)) {
            best = PivotKey{0u, 0u, 0x7fffffff};
            for (int i = j + lane; i < n; i += 32) pivot_offer(best, pivot_key(zabs(col[i]), i));
            best = pivot_reduce(best);
        }
        const int p = best.hi == 0u ? j : best.row;  // all-NaN column: keep the diagonal
        if (p != j) {
            for (int c = lane; c < n + nrhs; c += 32) {
                zc* cc = aug_col(L, X, n, c);
                const zc t = cc[j];
                cc[j] = cc[p];
                cc[p] = t;
            }
            __syncwarp();
        }
        const zc piv = col[j];
        if (is_zero(piv)) {
            if (lane == 0) sing_local[sys] = 1;
            for (int i = j + 1 + lane; i < n; i += 32) col[i] = zc{0.0, 0.0};
            __syncwarp();
            continue;
        }
        const zc inv = pivot_inverse(piv);
        const bool inv_ok = zfinite(inv);
        for (int i = j + 1 + lane; i < n; i += 32) col[i] = inv_ok ? col[i] * inv : zdiv(col[i], piv);
        // each lane updates the rows whose multipliers it just wrote; row j of the panel's columns was
        // settled by the swap above
        for (int c = j + 1; c < kend; ++c) {
            zc* cc = L + (long long)c * n;
            const zc u = cc[j];
            for (int i = j + 1 + lane; i < n; i += 32) cc[i] = zfms(col[i], u, cc[i]);
        }
        __syncwarp();
    }
    if (k0 + lane < kend) dinv[sys * n + k0 + lane] = pivot_inverse_refined(L[(long long)(k0 + lane) * (n + 1)]);
}

// The panel's row swaps on columns kend .. n+nrhs-1 (a warp per column), and with Solve the forward substitution of its
// rows with the panel's unit lower triangle: a lane per row, the solved entry broadcast. Solve takes twice the FP64
// instructions of a thread per column (half the lanes idle on average) but takes 14 us where that takes 90: for
// calls whose columns do not fill the GPU (kWarpColumnsLower).
template <bool Solve>
__global__ void __launch_bounds__(128) lu_swap_lower_kernel(int n, int nrhs, int batch, zc* lu, long long lu_stride, zc* x,
                                                            long long x_stride, int k0, int kend, const int* __restrict__ swaps,
                                                            int swap_stride, const int* __restrict__ skip, int skip_value) {
    const int cols = n + nrhs - kend, lane = threadIdx.x & 31;
    const long long idx = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (idx >= (long long)batch * cols) return;
    const long long sys = idx / cols;
    if (skip && skip[sys] == skip_value) return;
    const int c = kend + (int)(idx - sys * cols), w = kend - k0;
    zc* L = lu + sys * lu_stride;
    zc* cc = aug_col(L, x + sys * x_stride, n, c);
    const int* sw = swaps + sys * swap_stride;
    const int dst = sw[32 + lane];
    zc v = lane < w ? cc[sw[lane]] : zc{0.0, 0.0};
    zc moved{0.0, 0.0};
    if (dst >= 0) moved = cc[sw[64 + lane]];
    __syncwarp();
    if (dst >= 0) cc[dst] = moved;
    if (Solve) {
        const zc* l0 = L + (long long)k0 * n + k0 + lane;
#pragma unroll 8
        for (int q = 0; q + 1 < w; ++q) {
            const zc l = lane < w ? l0[(long long)q * n] : zc{0.0, 0.0};
            const zc xq{__shfl_sync(0xffffffffu, v.re, q), __shfl_sync(0xffffffffu, v.im, q)};
            const zc nv = zfms(l, xq, v);
            if (lane > q) v = nv;
        }
    }
    if (lane < w) cc[k0 + lane] = v;
}

// Rows r0 .. r1-1 (at most 32) of the right-hand sides: backward substitution with the diagonal block of U, a warp per
// column, a lane per row.
__global__ void __launch_bounds__(128) lu_upper_warp_kernel(int n, int nrhs, int batch, const zc* lu, long long lu_stride,
                                                            const zc* __restrict__ dinv, zc* x, long long x_stride, int r0, int r1,
                                                            const int* __restrict__ skip, int skip_value) {
    const long long idx = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (idx >= (long long)batch * nrhs) return;
    const long long sys = idx / nrhs;
    if (skip && skip[sys] == skip_value) return;
    const int c = (int)(idx - sys * nrhs), lane = threadIdx.x & 31, w = r1 - r0;
    const zc* U = lu + sys * lu_stride + (long long)r0 * n + r0 + lane;
    zc* xc = x + sys * x_stride + (long long)c * n + r0 + lane;
    zc v = lane < w ? *xc : zc{0.0, 0.0};
    const zc inv = lane < w ? dinv[sys * n + r0 + lane] : zc{1.0, 0.0};
    const bool inv_ok = zfinite(inv);
#pragma unroll 8
    for (int q = w - 1; q >= 0; --q) {
        const zc u = lane < q ? U[(long long)q * n] : zc{0.0, 0.0};
        const zc s = inv_ok ? v * inv : zdiv(v, U[(long long)lane * n]);
        const zc xq{__shfl_sync(0xffffffffu, s.re, q), __shfl_sync(0xffffffffu, s.im, q)};
        if (lane == q) v = xq;
        const zc nv = zfms(u, xq, v);
        if (lane < q) v = nv;
    }
    if (lane < w) *xc = v;
}

// Rows k0+1 .. kend-1 of columns kend .. n+nrhs-1: forward substitution with the panel's unit lower
// triangle, one thread per (system, column).
__global__ void lu_trsm_lower_kernel(int n, int nrhs, int batch, zc* lu, long long lu_stride, zc* x, long long x_stride,
                                     int k0, int kend, const int* __restrict__ skip, int skip_value) {
    const int cols = n + nrhs - kend;
    const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= (long long)batch * cols) return;
    const long long sys = idx / cols;
    if (skip && skip[sys] == skip_value) return;
    const int c = kend + (int)(idx - sys * cols);
    zc* L = lu + sys * lu_stride;
    zc* cc = aug_col(L, x + sys * x_stride, n, c);
    for (int r = k0 + 1; r < kend; ++r) {
        zc acc = cc[r];
        for (int q = k0; q < r; ++q) acc = zfms(L[(long long)q * n + r], cc[q], acc);
        cc[r] = acc;
    }
}

// Rows r0 .. r1-1 of the right-hand sides: backward substitution with the diagonal block of U.
__global__ void lu_trsm_upper_kernel(int n, int nrhs, int batch, const zc* lu, long long lu_stride,
                                     const zc* __restrict__ dinv, zc* x, long long x_stride, int r0, int r1,
                                     const int* __restrict__ skip, int skip_value) {
    const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= (long long)batch * nrhs) return;
    const long long sys = idx / nrhs;
    if (skip && skip[sys] == skip_value) return;
    const int c = (int)(idx - sys * nrhs);
    const zc* U = lu + sys * lu_stride;
    zc* xc = x + sys * x_stride + (long long)c * n;
    for (int r = r1 - 1; r >= r0; --r) {
        zc acc = xc[r];
        for (int q = r + 1; q < r1; ++q) acc = zfms(U[(long long)q * n + r], xc[q], acc);
        const zc inv = dinv[sys * n + r];
        xc[r] = zfinite(inv) ? acc * inv : zdiv(acc, U[(long long)r * n + r]);
    }
}

// a zero pivot in this call: the reference refuses to solve; the solution is reported as NaN
__global__ void lu_nan_fill_kernel(int n, int nrhs, int batch, zc* x, long long x_stride, const int* __restrict__ sing_local,
                                   int* __restrict__ singular) {
    const long long per = (long long)n * nrhs;
    const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= (long long)batch * per) return;
    const long long sys = idx / per;
    if (!sing_local[sys]) return;
    const double nan = __longlong_as_double(0x7ff8000000000000LL);
    x[sys * x_stride + (idx - sys * per)] = zc{nan, nan};
    if (idx - sys * per == 0) singular[sys] = 1;
}

// Batched complex GEMM: C = s_ab * (A B) + s_c * C0, one warp per 32 x COLS tile of C, lanes along rows (COLS 8, or 2 or
// 1 where more would leave schedulers without a warp: a step over k is 4 COLS FP64 instructions of 64 cycles).
// A: m x k (lda), B: k x n (ldb), C/C0: m x n (ldc); any stride may be 0 to broadcast one operand
// to the whole batch. s_ab, s_c in {-1, 0, 1}. C may alias C0 (each element is read then written by
// the same lane). The sums over k run in ascending order, as the reference's column GEMM adds
// (include/stablercwa/matrix.hpp:170-192); with COLS 1 and 2 the two products of each part have a sum of their own.
template <int COLS>
__global__ void __launch_bounds__(128) zgemm_kernel(int m, int n, int k, int batch, const zc* __restrict__ A, int lda,
                                                    long long a_stride, const zc* __restrict__ B, int ldb,
                                                    long long b_stride, const zc* C0, long long c0_stride, zc* C,
                                                    int ldc, long long c_stride, double s_ab, double s_c,
                                                    const int* __restrict__ skip, int skip_value, int tri) {
    const int tiles_m = (m + 31) / 32, tiles_n = (n + COLS - 1) / COLS;
    const long long warp = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const long long per = (long long)tiles_m * tiles_n;
    const long long sys = warp / per;
    if (sys >= batch) return;
    if (skip && skip[sys] == skip_value) return;
    const int t = (int)(warp - sys * per);
    const int tm = t % tiles_m, tn = t / tiles_m;
    const int lane = threadIdx.x & 31;
    const int row = tm * 32 + lane;
    const int c0 = tn * COLS;
    const int cols = min(COLS, n - c0);
    const zc* As = A + sys * a_stride;
    const zc* Bs = B + sys * b_stride;
    // with few columns the two products of a part are summed apart: half the chain, and half the growth of its error
    constexpr bool kApart = COLS <= 2;
    double ar[COLS], ai[COLS], br[COLS], bi[COLS];
#pragma unroll
    for (int j = 0; j < COLS; ++j) ar[j] = ai[j] = br[j] = bi[j] = 0.0;
    // a triangular factor: the k range that can hold nonzeros for this warp's rows / columns
    int p_begin = 0, p_end = k;
    if (tri == TRI_A_LOWER) p_end = min(k, tm * 32 + 32);
    else if (tri == TRI_A_UPPER) p_begin = tm * 32;
    else if (tri == TRI_B_UPPER) p_end = min(k, c0 + COLS);
    if (row < m) {
#pragma unroll 4
        for (int p = p_begin; p < p_end; ++p) {
            const zc av = As[(long long)p * lda + row];
#pragma unroll
            for (int j = 0; j < COLS; ++j) {
                if (j < cols) {
                    const zc bv = Bs[(long long)(c0 + j) * ldb + p];
                    if (kApart) {
                        ar[j] += av.re * bv.re;
                        ai[j] += av.re * bv.im;
                        br[j] -= av.im * bv.im;
                        bi[j] += av.im * bv.re;
                    } else {
                        ar[j] = ar[j] + av.re * bv.re - av.im * bv.im;
                        ai[j] = ai[j] + av.re * bv.im + av.im * bv.re;
                    }
                }
            }
        }
        const zc* C0s = C0 ? C0 + sys * c0_stride : nullptr;
        zc* Cs = C + sys * c_stride;
#pragma unroll
        for (int j = 0; j < COLS; ++j) {
            if (j < cols) {
                zc v = zc{s_ab * (ar[j] + br[j]), s_ab * (ai[j] + bi[j])};
                if (C0s && s_c != 0.0) {
                    const zc cv = C0s[(long long)(c0 + j) * ldc + row];
                    v = zc{s_c * cv.re + v.re, s_c * cv.im + v.im};
                }
                Cs[(long long)(c0 + j) * ldc + row] = v;
            }
        }
    }
}

// The same product without a triangular operand, a lane per element of C (U a lane, 32 apart in column-major order):
// for row counts of which 32-row tiles would leave lanes idle (9 rows: 28 % of them at work). Two 16-byte operands an
// element and step are far from the L1's rate beside four FP64 instructions of 64 cycles.
template <int U>
__global__ void __launch_bounds__(128) zgemm_flat_kernel(int m, int n, int k, int batch, const zc* __restrict__ A, int lda,
                                                         long long a_stride, const zc* __restrict__ B, int ldb, long long b_stride,
                                                         const zc* C0, long long c0_stride, zc* C, int ldc, long long c_stride,
                                                         double s_ab, double s_c, const int* __restrict__ skip, int skip_value) {
    const long long total = (long long)m * n, per = (total + 32 * U - 1) / (32 * U);
    const long long warp = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const long long sys = warp / per;
    if (sys >= batch) return;
    if (skip && skip[sys] == skip_value) return;
    const long long e0 = (warp - sys * per) * (32 * U) + (threadIdx.x & 31);
    const zc* As = A + sys * a_stride;
    const zc* Bs = B + sys * b_stride;
    const zc *pa[U], *pb[U];
    zc acc[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const long long e = min(e0 + 32 * u, total - 1), c = e / m;
        pa[u] = As + (e - c * m);
        pb[u] = Bs + c * ldb;
        acc[u] = zc{0.0, 0.0};
    }
#pragma unroll 2
    for (int p = 0; p < k; ++p)
#pragma unroll
        for (int u = 0; u < U; ++u) acc[u] = zmac(pa[u][(long long)p * lda], pb[u][p], acc[u]);
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const long long e = e0 + 32 * u;
        if (e >= total) break;
        const long long c = e / m, i = c * ldc + (e - c * m);
        zc v{s_ab * acc[u].re, s_ab * acc[u].im};
        if (C0 && s_c != 0.0) {
            const zc o = C0[sys * c0_stride + i];
            v = zc{s_c * o.re + v.re, s_c * o.im + v.im};
        }
        C[sys * c_stride + i] = v;
    }
}

// C = A B with A complex and B real (the eigenvectors Q Y of the Hermitian solver), zgemm_kernel's tiling:
// one warp per 32 x COLS tile of C, two fused multiply-adds per term.
template <int COLS>
__global__ void __launch_bounds__(128) zdgemm_kernel(int m, int n, int k, int batch, const zc* __restrict__ A, int lda,
                                                     long long a_stride, const double* __restrict__ B, int ldb,
                                                     long long b_stride, zc* __restrict__ C, int ldc, long long c_stride,
                                                     const int* __restrict__ skip, int skip_value) {
    const int tiles_m = (m + 31) / 32, tiles_n = (n + COLS - 1) / COLS;
    const long long warp = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const long long per = (long long)tiles_m * tiles_n;
    const long long sys = warp / per;
    if (sys >= batch) return;
    if (skip && skip[sys] == skip_value) return;
    const int t = (int)(warp - sys * per);
    const int tm = t % tiles_m, tn = t / tiles_m;
    const int row = tm * 32 + (threadIdx.x & 31);
    const int c0 = tn * COLS;
    const int cols = min(COLS, n - c0);
    if (row >= m) return;
    const zc* As = A + sys * a_stride;
    const double* Bs = B + sys * b_stride;
    double ar[COLS], ai[COLS];
#pragma unroll
    for (int j = 0; j < COLS; ++j) ar[j] = ai[j] = 0.0;
#pragma unroll 4
    for (int p = 0; p < k; ++p) {
        const zc av = As[(long long)p * lda + row];
#pragma unroll
        for (int j = 0; j < COLS; ++j) {
            if (j < cols) {
                const double bv = Bs[(long long)(c0 + j) * ldb + p];
                ar[j] = fma(av.re, bv, ar[j]);
                ai[j] = fma(av.im, bv, ai[j]);
            }
        }
    }
    zc* Cs = C + sys * c_stride;
#pragma unroll
    for (int j = 0; j < COLS; ++j)
        if (j < cols) Cs[(long long)(c0 + j) * ldc + row] = zc{ar[j], ai[j]};
}

}  // namespace rcwa_gb300
