// eig_fixed.cuh -- general complex eigensolver with the unitary transformations in 64-bit fixed point.
//
// The FP64 pipe of a GB300 issues 2 lanes a cycle per SM: one FP64 instruction of a warp takes 64 cycles of
// its scheduler, so a QR iteration in FP64 pays about 20 such instructions in a row for every Givens rotation
// (its dependent chain) and 12 per pair of entries it is applied to. The integer pipes issue 32-bit multiply-
// adds with 64-bit sums at more than ten times that rate and answer in a few cycles. Every quantity of the
// reduction is bounded: the rotations are unitary, and a unitary similarity keeps ||H||_2. So the matrix is
// scaled once by a power of two (N >= ||A||_2, the smaller of ||A||_F and sqrt(||A||_1 ||A||_inf), into
// [2^59, 2^60) units; the shifted H - t then stays below 2^61) and the whole iteration runs on integers. One
// unit is 2^-60 to 2^-59 N and a rounding half of it: FP64's for an entry of 2^-8 to 2^-7 N. Larger entries keep more
// bits than in FP64, smaller ones fewer; fix_range_kernel says for which matrices that matters and what happens to them.
//
//   rotation   G = [conj(q) s; -s q], q complex, s real, |q|^2 + s^2 = 1, held as round(c 2^60) in two limbs
//              c1 2^30 + c0 with c0 in [-2^29, 2^29) (zero-mean low limbs: the dropped low-by-low products
//              then have no bias)
//   entry      Y = y1 2^30 + y0, y0 in [0, 2^30)
//   product    C Y 2^-60 = c1 y1 + (c1 y0 + c0 y1) 2^-30 (+ c0 y0 2^-60, below half a unit, dropped): three
//              32 x 32 -> 64 multiply-adds; each output of a rotation is the sum of three products, nine
//              multiply-adds and one rounding
//   (q, s)     from 1 / sqrt(|x|^2 + sub^2): a float estimate corrected once to third order in integers
//
// Steps (one CTA per matrix for 1-3; eig_fixed.cu launches them):
//   1. Hessenberg form by Givens rotations: column k's entries are combined inside up to 16 row segments by
//      16 lanes at once, the segments' tops pairwise in log2 steps, then the rotations go to the rows (a lane
//      per column) and the columns (a lane per row). The subdiagonal comes out real.
//   2. Explicit single-shift QR (COMQR2's rotations, Wilkinson shift, deflation test). A sweep's left half runs in blocks of 32 columns: warp 0 holds the block's columns, a lane each,
//      forms the block's 32 rotations and applies them to its own columns as it goes, while the other warps
//      apply the previous block's rotations to the columns further right: one CTA barrier per block. The right
//      half is a lane per row.
//   3. Every rotation is logged.
//   4. Z: the log applied to an identity, a lane per row, the row in shared memory (fix_apply_kernel).
//   5. T from the reduced H (fix_triangle_kernel), its eigenvectors (fix_backsub_kernel) and V = Z X.
// Sums that a later sweep needs exactly (H - t) are exact: shifts are integers.
#pragma once

#include "eig.cuh"

namespace rcwa_gb300 {

struct __align__(16) lz {
    long long re, im;
};
struct FixRot {  // the limbs of q, s and of -Im q, -s
    int cr1, cr0, ci1, ci0, s1, s0, nc1, nc0, ns1, ns0;
};

constexpr int kFixSegs = 16;         // row segments of a column in the Hessenberg reduction
constexpr int kFixTilePitch = 33;    // a tile: 32 columns of 33 rows
constexpr int kFixTile = 32 * kFixTilePitch;
constexpr int kFixNormBits = 60;     // N < 2^60 units
constexpr int kFixEntry = 3;         // int4s of a rotation in shared memory (two in the log)

// log capacity in rotations: the reduction's (n^2 / 2 and a phase per segment) and 2.5 n^2 of the QR sweeps (a
// random matrix takes about 1.8 n^2, a grating layer's 1.0 n^2; a matrix that would need more is left to the
// FP64 kernels)
__host__ __device__ inline long long fix_reduce_capacity(int n) { return (long long)n * n / 2 + 17LL * n + 160; }
__host__ __device__ inline long long fix_log_capacity(int n) { return fix_reduce_capacity(n) + 5LL * n * n / 2; }
__host__ __device__ inline long long fix_table_capacity(int n) { return 8LL * n + 64; }
// shared memory of fix_schur_kernel: a tile a warp, one column's or sweep's rotations, the diagonal, the
// subdiagonal, the sweep's phase, reduction slots
__host__ __device__ inline size_t fix_schur_smem(int n, int warps) {
    return (size_t)warps * kFixTile * sizeof(lz) + (size_t)(n + kFixSegs) * kFixEntry * 16 + (size_t)n * (sizeof(lz) + 8) + 256;
}

__device__ __forceinline__ void fix_limbs(long long c, int& hi, int& lo) {
    lo = (int)((unsigned)c << 2) >> 2;
    hi = (int)(c >> 30) + (int)(((unsigned)c >> 29) & 1u);
}

// an entry's component as limbs y1 2^30 + y0 (|y| < 2^61)
struct FixLimb {
    int h, l;
};
__device__ __forceinline__ FixLimb fix_split(long long y) { return FixLimb{(int)(y >> 30), (int)((unsigned)y & 0x3fffffffu)}; }

// a x + b y + c z in the entries' units, coefficients (a1, a0) ...; z's terms last
__device__ __forceinline__ long long fix_dot3(int a1, int a0, const FixLimb& x, int b1, int b0, const FixLimb& y, int c1, int c0,
                                              const FixLimb& z) {
    long long u = fix_mad(a1, x.l, 1LL << 29);
    u = fix_mad(a0, x.h, u);
    u = fix_mad(b1, y.l, u);
    u = fix_mad(b0, y.h, u);
    long long h = fix_mad(a1, x.h, 0);
    h = fix_mad(b1, y.h, h);
    u = fix_mad(c1, z.l, u);
    u = fix_mad(c0, z.h, u);
    h = fix_mad(c1, z.h, h);
    return h + (u >> 30);
}

// oa = conj(q) a + s b, ob = q b - s a (Conj: q for conj(q) and the other way round); a is the value carried from
// rotation to rotation: its terms come last
template <bool Conj>
__device__ __forceinline__ void fix_pair(const FixRot& r, const lz& a, const lz& b, lz& oa, lz& ob) {
    const FixLimb ar = fix_split(a.re), ai = fix_split(a.im), br = fix_split(b.re), bi = fix_split(b.im);
    const int p1 = Conj ? r.nc1 : r.ci1, p0 = Conj ? r.nc0 : r.ci0, m1 = Conj ? r.ci1 : r.nc1, m0 = Conj ? r.ci0 : r.nc0;
    ob.re = fix_dot3(r.cr1, r.cr0, br, m1, m0, bi, r.ns1, r.ns0, ar);
    ob.im = fix_dot3(r.cr1, r.cr0, bi, p1, p0, br, r.ns1, r.ns0, ai);
    oa.re = fix_dot3(r.s1, r.s0, br, p1, p0, ai, r.cr1, r.cr0, ar);
    oa.im = fix_dot3(r.s1, r.s0, bi, m1, m0, ar, r.cr1, r.cr0, ai);
}
// conj(q) a (Conj: q a)
template <bool Conj>
__device__ __forceinline__ lz fix_phase(const FixRot& r, const lz& a) {
    const FixLimb ar = fix_split(a.re), ai = fix_split(a.im), o{0, 0};
    const int p1 = Conj ? r.nc1 : r.ci1, p0 = Conj ? r.nc0 : r.ci0, m1 = Conj ? r.ci1 : r.nc1, m0 = Conj ? r.ci0 : r.nc0;
    lz v;
    v.re = fix_dot3(0, 0, o, p1, p0, ai, r.cr1, r.cr0, ar);
    v.im = fix_dot3(0, 0, o, m1, m0, ar, r.cr1, r.cr0, ai);
    return v;
}

__device__ __forceinline__ float fix_rsqrt(float x) {
#ifdef __CUDA_ARCH__
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
#else
    return rsqrtf(x);
#endif
}

// the high words of |.| of three values (up to their signs' one unit), together
__device__ __forceinline__ int fix_tops(long long x, long long y, long long z) {
    const int a = (int)(x >> 32), b = (int)(y >> 32), c = (int)(z >> 32);
    return (a ^ (a >> 31)) | (b ^ (b >> 31)) | (c ^ (c >> 31));
}

// The rotation that takes (x, sub) to (nrm, 0): q = x / nrm, s = sub / nrm, nrm^2 = |x|^2 + sub^2, from components
// scaled so that the largest magnitude is in [2^60, 2^61).
__device__ __forceinline__ FixRot fix_rotation_scaled(long long xr, long long xi, long long sub) {
    const FixLimb a = fix_split(xr), b = fix_split(xi), c = fix_split(sub);
    // Q = (a^2 + b^2 + c^2) 2^-60, in [2^60, 3 2^62) (unsigned)
    const unsigned long long ll = (unsigned long long)((unsigned)a.l) * (unsigned)a.l + (unsigned long long)((unsigned)b.l) * (unsigned)b.l +
                                  (unsigned long long)((unsigned)c.l) * (unsigned)c.l;
    long long u = fix_mad(a.h, a.l, (1LL << 28) + (long long)(ll >> 31));
    u = fix_mad(b.h, b.l, u);
    u = fix_mad(c.h, c.l, u);
    long long Q = fix_mad(a.h, a.h, 0);
    Q = fix_mad(b.h, b.h, Q);
    Q = fix_mad(c.h, c.h, Q);
    Q += u >> 29;
    // y0 = 1 / sqrt(Q 2^-62) to about 22 bits, in units of 2^-29
    const unsigned y0 = (unsigned)(fix_rsqrt((float)(unsigned)((unsigned long long)Q >> 32)) * 17592186044416.0f);  // 2^44
    // e = 1 - q y0^2 exactly (Q Y0^2 against 2^120), then to 80 fractional bits; y = y0 (1 + e/2 + 3 e^2/8 + O(e^3))
    const unsigned long long P = (unsigned long long)y0 * y0;
    const unsigned long long lo = (unsigned long long)Q * P, hi = __umul64hi((unsigned long long)Q, P);
    const long long eh = (1LL << 56) - (long long)hi - (lo != 0 ? 1 : 0);
    const long long E = (long long)(((unsigned long long)eh << 24) | ((0ull - lo) >> 40));
    const int e32 = (int)(E >> 30);
    const long long D = ((E >> 1) + ((3 * fix_mad(e32, e32, 0)) >> 23) + (1 << 17)) >> 18;  // 62 fractional bits
    const int d1 = (int)(D >> 21), d0 = (int)((unsigned)D & 0x1fffffu);
    const long long y = ((long long)y0 << 30) + (fix_mad((int)y0, d1, (fix_mad((int)y0, d0, 0) >> 21) + (1 << 10)) >> 11);  // 59 fractional bits
    const FixLimb Y = fix_split(y);
    const auto scale = [&](const FixLimb& x) {  // x y: 60 fractional bits
        // (with the product of the low limbs: without its mean q and s came out a quarter of a unit low, |q|^2 + s^2
        // below one, and the QL iteration, whose diagonal takes that as an addition, moved every small eigenvalue up)
        long long v = fix_mad(x.h, Y.l, (long long)(1 << 29));
        v = fix_mad(x.l, Y.h, v) + (fix_mad(x.l, Y.l, 0) >> 30);
        return fix_mad(x.h, Y.h, v >> 30);
    };
    FixRot r;
    fix_limbs(scale(a), r.cr1, r.cr0);
    fix_limbs(scale(b), r.ci1, r.ci0);
    fix_limbs(scale(c), r.s1, r.s0);
    r.nc1 = -r.ci1;
    r.nc0 = -r.ci0;
    r.ns1 = -r.s1;
    r.ns0 = -r.s0;
    return r;
}

// The same from components below 2^61; the identity for x = sub = 0.
__device__ __forceinline__ FixRot fix_rotation(long long xr, long long xi, long long sub) {
    int h = fix_tops(xr, xi, sub);
    if (h == 0) {  // all of them below 2^32 units
        if ((xr | xi | sub) == 0) xr = 1;
        xr <<= 27;
        xi <<= 27;
        sub <<= 27;
        h = fix_tops(xr, xi, sub);
        if (h == 0) {
            xr <<= 27;
            xi <<= 27;
            sub <<= 27;
            h = fix_tops(xr, xi, sub);
        }
    }
    const int sh = __clz(h) - 3;  // the largest into [2^60, 2^61)
    return fix_rotation_scaled(xr << sh, xi << sh, sub << sh);
}

// a rotation in shared memory (kFixEntry int4s) and in the log (two)
__device__ __forceinline__ void fix_put(int4* p, const FixRot& r) {
    p[0] = make_int4(r.cr1, r.cr0, r.s1, r.s0);
    p[1] = make_int4(r.ci1, r.ci0, r.nc1, r.nc0);
    p[2] = make_int4(r.ns1, r.ns0, 0, 0);
}
__device__ __forceinline__ FixRot fix_get(const int4* p) {
    const int4 u = p[0], v = p[1];
    const int2 w = *reinterpret_cast<const int2*>(p + 2);
    return FixRot{u.x, u.y, v.x, v.y, u.z, u.w, v.z, v.w, w.x, w.y};
}
__device__ __forceinline__ FixRot fix_log_get(const int4& u, const int4& v) {
    return FixRot{u.x, u.y, v.x, v.y, u.z, u.w, v.z, v.w, -u.z, -u.w};
}

// x 2^(-e) in units (x finite, |x 2^-e| < 2^62), to nearest
__device__ __forceinline__ long long fix_from_double(double x, int e) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(x);
    const int be = (int)((b >> 52) & 0x7FF);
    if (be == 0) return 0;  // zero; a subnormal entry is below the resolution of any scale reached here
    const unsigned long long mant = (b & 0xFFFFFFFFFFFFFull) | (1ull << 52);
    const int sh = be - 1075 - e;
    unsigned long long m = 0;
    if (sh >= 0) {
        m = sh < 10 ? mant << sh : 0;
    } else if (sh > -54) {
        m = (mant + (1ull << (-sh - 1))) >> -sh;
    }
    return (b >> 63) ? -(long long)m : (long long)m;
}

// the segments of column k's m = n - 1 - k entries below the diagonal: `len` rows each (the last shorter)
__device__ __forceinline__ int fix_seg_len(int m) { return max(2, (m + kFixSegs - 1) / kFixSegs); }

// 16 bytes from global to shared memory without a register in between; fix_copy_wait for the calling thread's
__device__ __forceinline__ void fix_copy16(lz* dst, const lz* src) {
#ifdef __CUDA_ARCH__
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
#else
    *dst = *src;
#endif
}
__device__ __forceinline__ void fix_copy_wait() {
#ifdef __CUDA_ARCH__
    asm volatile("cp.async.wait_all;" ::: "memory");
#endif
}

// Rows r0 .. r0 + rows - 1 (at most 32) of columns c0 .. c0 + nc - 1 into the warp's tile, every copy in flight at
// once, and back.
__device__ __forceinline__ void fix_tile_load(int n, const lz* H, lz* tile, int r0, int rows, int c0, int nc) {
    const int lane = threadIdx.x & 31;
    const lz* src = H + (long long)c0 * n + r0 + lane;
    if (lane < rows)
        for (int c = 0; c < nc; ++c) fix_copy16(tile + c * kFixTilePitch + lane, src + (long long)c * n);
    fix_copy_wait();
    __syncwarp();
}
__device__ __forceinline__ void fix_tile_store(int n, lz* H, const lz* tile, int r0, int rows, int c0, int nc) {
    const int lane = threadIdx.x & 31;
    __syncwarp();
    lz* dst = H + (long long)c0 * n + r0 + lane;
    if (lane < rows) {
#pragma unroll 4
        for (int c = 0; c < nc; ++c) dst[(long long)c * n] = tile[c * kFixTilePitch + lane];
    }
    __syncwarp();
}

// The rotations r0 + 1 .. r0 + cnt, cnt <= 32 (rows i - 1, i; rots[kFixEntry i] in shared memory) applied to rows
// r0 .. r0 + cnt of columns c0 .. c0 + nc - 1, a lane per column; returns the lane's row r0 + cnt, which is not
// stored.
__device__ __forceinline__ lz fix_left_block(int n, lz* H, lz* tile, const int4* rots, int r0, int cnt, int c0, int nc) {
    const int lane = threadIdx.x & 31;
    lz y{0, 0};
    if (lane < nc) y = H[(long long)(c0 + lane) * n + r0 + cnt];
    fix_tile_load(n, H, tile, r0, cnt, c0, nc);
    if (lane < nc) {
        lz* t = tile + lane * kFixTilePitch;
        t[cnt] = y;
        y = t[0];
        lz z = t[1];
#pragma unroll 2
        for (int i = 1; i <= cnt; ++i) {
            const lz zn = t[min(i + 1, cnt)];
            lz a, b;
            fix_pair<false>(fix_get(rots + kFixEntry * (r0 + i)), y, z, a, b);
            t[i - 1] = a;
            y = b;
            z = zn;
        }
    }
    fix_tile_store(n, H, tile, r0, cnt, c0, nc);
    return y;
}

// ---- which matrices the fixed-point kernels may take
//
// One unit of 2^-59 N or less is lost wherever an entry is held: a row of size m keeps 2^-59 N / m of itself, however small
// m is. FP64 loses more where its reflectors or shifts mix such a row with those of size N, as on a layer matrix
// Kx^2 - [[eps]], whose centre is 2^-16 of N and tied to the rest by the profile's harmonics; where they do not it keeps
// 2^-53 of the row, and such matrices stay with the FP64 kernels:
//   - general solver: matrices whose last row or column is 2^-7 below the largest (graded downwards, or a small block last:
//     deflated before a large shift has passed over them). Last rows without entries left of the diagonal deflate before
//     there is a shift: a small diagonal entry in one of them counts, and past them the last row or column of the block
//     that is left; upper triangular matrices are nothing else. A layer's last order is one of its largest (2^-4 of it at
//     grazing incidence on a wide period), with entries to its left.
//   - Hermitian solver: rows 2^-7 below the largest that nothing ties to larger ones (diagonal matrices, separate blocks),
//     in which the entries towards rows 2^3 larger are below 2^-40 of the row, or, 2^-14 below the largest, those
//     towards rows 2^7 larger below 2^-16; and tridiagonal matrices with a row 2^-7 below the largest. The centre rows of layers,
//     contrasts of a few percent among them, are tied by 2^-12 and more, for periods of 0.1 to 10 wavelengths.
// Largest relative error of an eigenvalue at order 30 against 60 digits, FP64 / fixed point: diag(1 .. 1e-20) 0 / 1; a
// block of 1e-4 of the other 3e-15 / 3e-12 (last, general), 2e-14 / 1e-12 (Hermitian); rows and columns graded downwards
// over 1e-5 each, general 4e-14 / 2e-7, over 1e-2.1 2e-14 / 4e-13; triangular 0 / 6e-6; tridiagonal graded over 1e-4
// 8e-16 / 5e-11. What stays here: layers 2e-13 to 1e-11 / 2e-14 to 7e-13; graded upwards over 1e-5, general 4e-7 / 4e-8,
// Hermitian 4e-7 / 9e-8; Hermitian graded downwards over 1e-5 8e-8 / 3e-8; a small block first, general, 8e-12 / 2e-12.
// The magnitudes are the upper words of the larger component (a lower word alone counts as the smallest).
constexpr int kFixRangeThreads = 512;
constexpr int kFixRangeSmall = 7 << 20, kFixRangeFar = 14 << 20, kFixRangeTie = 16 << 20;
constexpr int kFixRangeLarger = 3 << 20, kFixRangeUntied = 40 << 20;
__host__ __device__ inline size_t fix_range_smem(int n) { return ((size_t)2 * n + 2) * sizeof(int); }

__device__ __forceinline__ int fix_magnitude(const zc& z) {
    const unsigned long long x = (unsigned long long)__double_as_longlong(z.re) << 1, y = (unsigned long long)__double_as_longlong(z.im) << 1;
    const unsigned long long m = x > y ? x : y;
    return m == 0 ? 0 : max((int)(m >> 33), 1);
}

// the largest of a warp's values (none negative)
__device__ __forceinline__ int fix_warp_max(int v) {
#ifdef __CUDA_ARCH__
    return (int)__reduce_max_sync(0xffffffffu, (unsigned)v);
#else
    for (int o = 16; o > 0; o >>= 1) v = max(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
#endif
}

__device__ __forceinline__ void fix_shared_max(int* p, int v) {
#ifdef __CUDA_ARCH__
    atomicMax(p, v);
#else
    *p = max(*p, v);
#endif
}

// Hermitian matrices; status[b]: `other` for one that the FP64 kernels keep, else 0. A CTA per matrix, which it reads once (a warp takes
// 32 rows of eight columns at a time, all loads in flight); then a warp for every small row or column. Latency bounds it
// for one matrix (order 121: 11 us cold; with 128 threads, 32 rows and all columns a warp, 65), the memory for 4096 (0.18 ms).
static __global__ void __launch_bounds__(kFixRangeThreads) fix_range_kernel(int n, int batch, const zc* __restrict__ a_in,
                                                                            long long a_stride, int* __restrict__ status, int other) {
    RCWA_DYN_SMEM(int, fix_rg);
    const long long gid = blockIdx.x;
    if (gid >= batch) return;
    const zc* A = a_in + gid * a_stride;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nthr = blockDim.x, nw = nthr >> 5;
    int *rs = fix_rg, *cs = rs + n, *flags = cs + n;  // largest of each row and column; [0] beside the band, [1] the FP64 kernels'
    for (int i = tid; i < 2 * n + 2; i += nthr) fix_rg[i] = 0;
    __syncthreads();
    bool outside = false;
    const int chunks = (n + 31) / 32, items = chunks * ((n + 7) / 8);
    for (int q = warp; q < items; q += nw) {
        const int r = 32 * (q % chunks) + lane, c0 = 8 * (q / chunks);
        const bool in = r < n;
        const zc* a = A + (long long)c0 * n + (in ? r : n - 1);
        int v[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) v[u] = fix_magnitude(a[(long long)min(u, n - 1 - c0) * n]);  // the last column again
        int m = 0, col = 0;
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            const int c = min(c0 + u, n - 1);
            m = max(m, v[u]);
            outside |= in && v[u] != 0 && (c + 1 < r || r + 1 < c);
            const int w = fix_warp_max(in ? v[u] : 0);
            if (lane == u) col = w;
        }
        if (in) fix_shared_max(rs + r, m);
        if (lane < 8) fix_shared_max(cs + min(c0 + lane, n - 1), col);
    }
    if (outside) flags[0] = 1;
    __syncthreads();
    int top = 0, high = 0;  // the largest, and 2^31 - 1 less the smallest that is not zero
    for (int i = lane; i < n; i += 32) {
        if (warp == 0) rs[i] = max(rs[i], cs[i]);
        const int m = max(rs[i], cs[i]);
        top = max(top, m);
        if (m) high = max(high, 0x7fffffff - m);
    }
    top = fix_warp_max(top);
    const int low = 0x7fffffff - fix_warp_max(high);
    __syncthreads();
    bool keep = false;
    if (top != 0 && top < 0x7ff00000 && low + kFixRangeSmall <= top) {  // zero and non-finite matrices are the solver's own to leave
        keep = !flags[0];
        for (int i = warp; i < n; i += nw) {
            const int m = rs[i];
            if (m == 0 || m + kFixRangeSmall > top) continue;
            const bool far = m + kFixRangeFar <= top;
            int tie = 0;
            for (int k = lane; k < n; k += 32)
                if (rs[k] >= m + (far ? kFixRangeSmall : kFixRangeLarger))
                    tie = max(tie, max(fix_magnitude(A[(long long)k * n + i]), fix_magnitude(A[(long long)i * n + k])));
            keep |= fix_warp_max(tie) + (far ? kFixRangeTie : kFixRangeUntied) <= m;
        }
    }
    if (keep) flags[1] = 1;
    __syncthreads();
    if (tid == 0) status[gid] = flags[1] ? other : 0;
}

// The general solver's, by all threads of its CTA (flags: 4 slots a warp), in its own kernel: as a launch of its own it took 0.9 %
// of a sweep of small batches (two gratings, 128 samples of order 61: 25.85 to 26.07 ms), so 25.85.
__device__ __forceinline__ bool fix_keeps_fp64(int n, const zc* __restrict__ A, int* flags) {
    const int tid = threadIdx.x, nthr = blockDim.x, nw = nthr >> 5;
    int v[4] = {0, 0, 0, 0};  // the largest, in the last row, in the last column; the rows up to the last with an entry left of its diagonal
    const auto all = [&] {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int m = fix_warp_max(v[q]);
            if ((tid & 31) == 0) flags[4 * (tid >> 5) + q] = m;
        }
        __syncthreads();
        for (int w = 0; w < nw; ++w)
#pragma unroll
            for (int q = 0; q < 4; ++q) v[q] = max(v[q], flags[4 * w + q]);
        __syncthreads();
    };
    for (int r = tid; r < n; r += nthr)
#pragma unroll 8
        for (int c = 0; c < n; ++c) {
            const int m = fix_magnitude(A[(long long)c * n + r]);
            v[0] = max(v[0], m);
            if (r == n - 1) v[1] = max(v[1], m);
            if (c == n - 1) v[2] = max(v[2], m);
            if (r > c && m) v[3] = r + 1;
        }
    all();
    const int p = v[3], small = v[0] - kFixRangeSmall;
    if (p == 0) return true;
    if (p < n) {
        // the rows from p on deflate before there is a shift: their diagonal entries, then the block before them
        v[1] = v[2] = v[3] = 0;
        for (int i = tid; i < n; i += nthr) {
            if (i < p) {
                v[1] = max(v[1], fix_magnitude(A[(long long)i * n + p - 1]));
                v[2] = max(v[2], fix_magnitude(A[(long long)(p - 1) * n + i]));
            } else if (fix_magnitude(A[(long long)i * (n + 1)]) <= small) {
                v[3] = 1;
            }
        }
        all();
        if (v[3]) return true;
    }
    return min(v[1], v[2]) <= small;
}

constexpr int kFixBatch = 6;  // columns whose entries a row's lane holds at once, and as many on their way

// What bounds it: latency. 456 matrices of order 121 take 36.3 ms with 6 warps an SM, 0.9 instructions a cycle and no pipe
// above 22 %; the warps wait at the barriers (3.3 of their stalls an issue, next the multiply-adds' own 1.3) for the one that
// forms a block's rotations.
//
// Schur reduction of one matrix; with Herm only step 1, on the Hermitian part (A + A^H) / 2: the reduced matrix is
// real symmetric tridiagonal, its d and e go where the QL kernel reads them. H: n x n lz (column-major, global). log: rotations (two int4 each), table:
// (l, en, phase) per sweep in int4. w: eigenvalues in deflation order. status: 0 done, 1 left to the FP64
// kernels (non-finite input, no convergence, log full; other[b] set, or `check` and fix_keeps_fp64). head: the
// number of sweeps and the exponent of the unit.
template <bool Herm>
__global__ void fix_schur_kernel(int n, int batch, const zc* __restrict__ a_in, long long a_stride, zc* __restrict__ w_out,
                                        lz* __restrict__ h_ws, long long h_stride, int4* __restrict__ log_all, long long log_stride,
                                        int4* __restrict__ table_all, int* __restrict__ head, int* __restrict__ status,
                                        int* __restrict__ done, int* __restrict__ info, const int* __restrict__ other = nullptr,
                                        bool check = false) {
    RCWA_DYN_SMEM(lz, fix_sm);
    const long long gid = blockIdx.x;
    if (gid >= batch) return;
    if (other && other[gid]) {
        if (threadIdx.x == 0) status[gid] = 1;
        return;
    }
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nthr = blockDim.x, nw = nthr >> 5;
    lz* tiles = fix_sm;
    lz* tile = tiles + (long long)warp * kFixTile;
    int4* rots = reinterpret_cast<int4*>(tiles + (long long)nw * kFixTile);  // kFixEntry (n + kFixSegs)
    int4* phase = rots + kFixEntry * (n + kFixSegs);                         // kFixEntry
    lz* dg = reinterpret_cast<lz*>(phase + kFixEntry);                              // n
    long long* sub = reinterpret_cast<long long*>(dg + n);                  // n
    int* flags = reinterpret_cast<int*>(sub + n);                           // 48 reduction slots, [48] the phase flag
    const zc* A = a_in + gid * a_stride;
    lz* H = h_ws + gid * h_stride;
    int4* log = log_all + gid * log_stride;
    int4* table = table_all + gid * fix_table_capacity(n);
    const long long nn = (long long)n * n;
    const lz zero{0, 0};

    if constexpr (!Herm) {
        if (check && fix_keeps_fp64(n, A, flags)) {
            if (tid == 0) {
                status[gid] = 1;
                done[gid] = 0;
            }
            return;
        }
    }
    // ---- scale: the largest exponent, then N (sums in a fixed order)
    int top = 0;
    for (long long i = tid; i < nn; i += nthr) {
        const zc z = A[i];
        top = max(top, max((int)((__double_as_longlong(z.re) >> 52) & 0x7FF), (int)((__double_as_longlong(z.im) >> 52) & 0x7FF)));
    }
    for (int o = 16; o > 0; o >>= 1) top = max(top, __shfl_xor_sync(0xffffffffu, top, o));
    if (lane == 0) flags[warp] = top;
    __syncthreads();
    for (int q = 0; q < nw; ++q) top = max(top, flags[q]);
    __syncthreads();
    // outside a range that keeps every power of two used here a normal double (zero matrices and non-finite
    // entries included) the FP64 kernels take the matrix
    if (top < 200 || top > 1900) {
        if (tid == 0) {
            status[gid] = 1;
            if (!Herm) done[gid] = 0;
        }
        return;
    }
    // in float, relative to 2^(top - 1023): the row sums and squares a lane per row, the column sums a warp each
    float ss = 0.0f, rmax = 0.0f, cmax = 0.0f;
    {
        const double scl = __longlong_as_double((long long)(2046 - top) << 52);  // the largest component into [1, 2)
        for (int r = tid; r < n; r += nthr) {
            float rs = 0.0f;
            for (int c = 0; c < n; ++c) {
                const zc z = A[(long long)c * n + r];
                const float x = (float)(z.re * scl), y = (float)(z.im * scl), q = x * x + y * y;
                ss += q;
                rs += sqrtf(q);
            }
            rmax = fmaxf(rmax, rs);
        }
        for (int c = warp; c < n; c += nw) {
            float cs = 0.0f;
            for (int r = lane; r < n; r += 32) {
                const zc z = A[(long long)c * n + r];
                const float x = (float)(z.re * scl), y = (float)(z.im * scl);
                cs += sqrtf(x * x + y * y);
            }
            for (int o = 16; o > 0; o >>= 1) cs += __shfl_xor_sync(0xffffffffu, cs, o);
            cmax = fmaxf(cmax, cs);
        }
        for (int o = 16; o > 0; o >>= 1) {
            ss += __shfl_xor_sync(0xffffffffu, ss, o);
            rmax = fmaxf(rmax, __shfl_xor_sync(0xffffffffu, rmax, o));
        }
        if (lane == 0) {
            flags[warp] = __float_as_int(ss);
            flags[16 + warp] = __float_as_int(rmax);
            flags[32 + warp] = __float_as_int(cmax);
        }
        __syncthreads();
        ss = 0.0f;
        for (int q = 0; q < nw; ++q) {
            ss += __int_as_float(flags[q]);
            rmax = fmaxf(rmax, __int_as_float(flags[16 + q]));
            cmax = fmaxf(cmax, __int_as_float(flags[32 + q]));
        }
        __syncthreads();
    }
    // N = 2^(top - 1023) min(..) < 2^(e2 + kFixNormBits)
    const int e2 = ((__float_as_int(fminf(sqrtf(ss), sqrtf(rmax * cmax)) * 1.001f) >> 23) & 0xff) - 127 + 1 + (top - 1023) - kFixNormBits;
    if constexpr (Herm) {
        for (long long i = tid; i < nn; i += nthr) {
            const int c = (int)(i / n), r = (int)(i - (long long)c * n);
            const zc x = A[i], y = A[(long long)r * n + c];
            H[i] = lz{fix_from_double(0.5 * (x.re + y.re), e2), fix_from_double(0.5 * (x.im - y.im), e2)};
        }
    } else {
        for (long long i = tid; i < nn; i += nthr) H[i] = lz{fix_from_double(A[i].re, e2), fix_from_double(A[i].im, e2)};
    }
    __syncthreads();

    // ---- Hessenberg form
    long long pos = 0;
    for (int k = 0; k + 1 < n; ++k) {
        const int m = n - 1 - k, len = fix_seg_len(m), ns = (m + len - 1) / len, top_row = k + 1;
        lz* ck = H + (long long)k * n;
        // entries of this column: per segment (bottom up) a phase and its rotations, then the tree
        const long long tree0 = pos + m;  // m - ns rotations and ns phases before the tree
        if (warp == 0) {
            long long carry = 0;
            if (lane < ns) {
                const int t0 = top_row + lane * len, t1 = min(t0 + len, n);
                long long p = pos + (long long)lane * len;
                lz x = ck[t1 - 1];
                FixRot r = fix_rotation(x.re, x.im, 0);
                fix_put(rots + kFixEntry * (p - pos), r);
                ++p;
                carry = fix_phase<false>(r, x).re;
                for (int i = t1 - 2; i >= t0; --i, ++p) {
                    x = ck[i];
                    r = fix_rotation(x.re, x.im, carry);
                    fix_put(rots + kFixEntry * (p - pos), r);
                    lz oa, ob;
                    fix_pair<false>(r, x, lz{carry, 0}, oa, ob);
                    carry = oa.re;
                }
            }
            __syncwarp();
            long long p = tree0;
            for (int d = 1; d < ns; d *= 2) {
                const long long other = __shfl_down_sync(0xffffffffu, carry, d);
                const int pairs = (ns - d + 2 * d - 1) / (2 * d);  // lanes 0, 2d, 4d, .. with lane + d < ns
                if (lane % (2 * d) == 0 && lane + d < ns) {
                    const FixRot r = fix_rotation(carry, 0, other);
                    const long long q = p + lane / (2 * d);
                    fix_put(rots + kFixEntry * (q - pos), r);
                    lz oa, ob;
                    fix_pair<false>(r, lz{carry, 0}, lz{other, 0}, oa, ob);
                    carry = oa.re;
                }
                p += pairs;
            }
            if (lane == 0) sub[k + 1] = carry;
        }
        __syncthreads();
        const int nent = m + ns - 1;
        for (int i = tid; i < 2 * nent; i += nthr) log[2 * pos + i] = rots[kFixEntry * (i >> 1) + (i & 1)];
        // rows, columns k + 1 ..: a lane per column
        const int per = max(1, 32 / len);  // segments per tile
        for (int g0 = k + 1 + 32 * warp; g0 < n; g0 += 32 * nw) {
            const int nc = min(32, n - g0);
            for (int s0 = 0; s0 < ns; s0 += per) {
                const int r0 = top_row + s0 * len, rows = min(min(per, ns - s0) * len, n - r0);
                fix_tile_load(n, H, tile, r0, rows, g0, nc);
                if (lane < nc) {
                    lz* t = tile + lane * kFixTilePitch - r0;
                    for (int sg = s0; sg < min(s0 + per, ns); ++sg) {
                        const int t0 = top_row + sg * len, t1 = min(t0 + len, n);
                        const int4* e = rots + kFixEntry * (sg * len);
                        lz y = fix_phase<false>(fix_get(e), t[t1 - 1]);
                        lz x = t[max(t1 - 2, t0)];
                        for (int i = t1 - 2; i >= t0; --i) {
                            const lz xn = t[max(i - 1, t0)];
                            e += kFixEntry;
                            lz oa, ob;
                            fix_pair<false>(fix_get(e), x, y, oa, ob);
                            t[i + 1] = ob;
                            y = oa;
                            x = xn;
                        }
                        t[t0] = y;
                    }
                }
                fix_tile_store(n, H, tile, r0, rows, g0, nc);
            }
            // the tree, on the segments' tops
            if (lane < nc) {
                lz* hc = H + (long long)(g0 + lane) * n + top_row;
                lz* t = tile + lane * kFixTilePitch;
                for (int sg = 0; sg < ns; ++sg) fix_copy16(t + sg, hc + sg * len);
                fix_copy_wait();
                const int4* e = rots + kFixEntry * m;
                for (int d = 1; d < ns; d *= 2)
                    for (int sg = 0; sg + d < ns; sg += 2 * d, e += kFixEntry) {
                        lz oa, ob;
                        fix_pair<false>(fix_get(e), t[sg], t[sg + d], oa, ob);
                        t[sg] = oa;
                        t[sg + d] = ob;
                    }
                for (int sg = 0; sg < ns; ++sg) hc[sg * len] = t[sg];
            }
            __syncwarp();
        }
        __syncthreads();
        // columns k + 1 .., every row: a lane per row
        for (int r = tid; r < n; r += nthr) {
            lz* hr = H + r;
            // the segments' entries from the last column down, kFixBatch of them in registers and the next
            // batch on its way: one continuous run over columns n - 1 .. k + 1 within each segment
            lz* t = tile + lane * kFixTilePitch;  // the segments' tops
            for (int sg = 0; sg < ns; ++sg) {
                const int t0 = top_row + sg * len, t1 = min(t0 + len, n);
                const int4* e = rots + kFixEntry * (sg * len);
                lz buf[kFixBatch], nxt[kFixBatch];
                lz y = hr[(long long)(t1 - 1) * n];
#pragma unroll
                for (int u = 0; u < kFixBatch; ++u) buf[u] = hr[(long long)max(t1 - 2 - u, t0) * n];
                y = fix_phase<true>(fix_get(e), y);
                for (int i = t1 - 2; i >= t0; i -= kFixBatch) {
#pragma unroll
                    for (int u = 0; u < kFixBatch; ++u) nxt[u] = hr[(long long)max(i - kFixBatch - u, t0) * n];
#pragma unroll
                    for (int u = 0; u < kFixBatch; ++u)
                        if (i - u >= t0) {
                            e += kFixEntry;
                            lz oa, ob;
                            fix_pair<true>(fix_get(e), buf[u], y, oa, ob);
                            hr[(long long)(i - u + 1) * n] = ob;
                            y = oa;
                        }
#pragma unroll
                    for (int u = 0; u < kFixBatch; ++u) buf[u] = nxt[u];
                }
                t[sg] = y;
            }
            const int4* e = rots + kFixEntry * m;
            for (int d = 1; d < ns; d *= 2)
                for (int sg = 0; sg + d < ns; sg += 2 * d, e += kFixEntry) {
                    lz oa, ob;
                    fix_pair<true>(fix_get(e), t[sg], t[sg + d], oa, ob);
                    t[sg] = oa;
                    t[sg + d] = ob;
                }
            for (int sg = 0; sg < ns; ++sg) hr[(long long)(top_row + sg * len) * n] = t[sg];
        }
        pos += nent;
        __syncthreads();
    }
    for (int i = tid; i < n; i += nthr) dg[i] = H[(long long)i * n + i];
    if (tid == 0) sub[0] = 0;
    __syncthreads();

    if constexpr (Herm) {
        const double unit = __longlong_as_double((long long)(e2 + 1023) << 52);
        double* d = reinterpret_cast<double*>(H + 2 * nn);
        for (int i = tid; i < n; i += nthr) {
            d[i] = (double)dg[i].re * unit;
            d[n + i] = i + 1 < n ? (double)sub[i + 1] * unit : 0.0;
        }
        if (tid == 0) {
            head[2 * gid] = 0;
            status[gid] = 0;
        }
        return;
    }

    // ---- shifted QR
    const long long log_cap = log_stride / 2, tab_cap = fix_table_capacity(n);
    const double unit = __longlong_as_double((long long)(e2 + 1023) << 52);
    lz t{0, 0};
    int en = n - 1, its = 0, sweeps = 0, fail = 0;
    while (en >= 0) {
        int l = 0;
        for (int base = en; base >= 1; base -= 32) {
            const int c = base - lane;
            bool ok = false;
            if (c >= 1) {
                const long long s = sub[c] < 0 ? -sub[c] : sub[c];
                const lz p = dg[c - 1], q = dg[c];
                const unsigned long long size = (unsigned long long)((p.re < 0 ? -p.re : p.re) + (p.im < 0 ? -p.im : p.im)) +
                                                (unsigned long long)((q.re < 0 ? -q.re : q.re) + (q.im < 0 ? -q.im : q.im));
                // eps (|h(c-1, c-1)| + |h(c, c)|), or two units (at most 2^-58 N)
                ok = s <= 2 || (unsigned long long)s <= (size >> 52);
            }
            const unsigned bits = __ballot_sync(0xffffffffu, ok);
            if (bits) {
                l = base - (__ffs(bits) - 1);
                break;
            }
        }
        if (l == en) {
            if (tid == 0) w_out[gid * n + en] = zc{(double)(dg[en].re + t.re) * unit, (double)(dg[en].im + t.im) * unit};
            --en;
            its = 0;
            continue;
        }
        if (its == 30 || pos + (en - l) + 129 > log_cap || sweeps >= tab_cap) {
            fail = 1;
            break;
        }
        // Wilkinson shift: d - x / (y + sqrt(y^2 + x)), y = (a - d) / 2, x = b c; the correction in float. The
        // tenth and twentieth iterations take the exceptional shift |h(en, en-1)| + |h(en-1, en-2)| where the
        // shifted matrix then still fits the scale (|t| < 2^60 units).
        lz s = dg[en];
        const long long ex = (sub[en] < 0 ? -sub[en] : sub[en]) + (en >= 2 ? (sub[en - 1] < 0 ? -sub[en - 1] : sub[en - 1]) : 0);
        if ((its == 10 || its == 20) && (t.re < 0 ? -t.re : t.re) + (t.im < 0 ? -t.im : t.im) + ex < (1LL << 60)) {
            s = lz{ex, 0};
        } else {
            const lz pa = dg[en - 1], pb = H[(long long)en * n + en - 1];
            const float k = 0x1p-60f;
            const float yr = (float)((pa.re - s.re) >> 1) * k, yi = (float)((pa.im - s.im) >> 1) * k;
            const float c = (float)sub[en] * k, xr = (float)pb.re * k * c, xi = (float)pb.im * k * c;
            if (xr != 0.0f || xi != 0.0f) {
                const float zr = yr * yr - yi * yi + xr, zi = 2.0f * yr * yi + xi;
                const float mod = sqrtf(zr * zr + zi * zi);
                float rr, ri;
                if (zr >= 0.0f) {
                    rr = sqrtf(0.5f * (mod + zr));
                    ri = rr > 0.0f ? 0.5f * zi / rr : 0.0f;
                } else {
                    ri = sqrtf(0.5f * (mod - zr));
                    rr = ri > 0.0f ? 0.5f * zi / ri : 0.0f;
                }
                if (yr * rr + yi * ri < 0.0f) {
                    rr = -rr;
                    ri = -ri;
                }
                const float dr = yr + rr, di = yi + ri, dd = dr * dr + di * di;
                if (dd > 1e-37f) {
                    const float cr = (xr * dr + xi * di) / dd, ci = (xi * dr - xr * di) / dd;
                    s.re -= (long long)(cr * 0x1p60f);
                    s.im -= (long long)(ci * 0x1p60f);
                }
            }
        }
        t.re += s.re;
        t.im += s.im;
        ++its;
        __syncthreads();
        for (int r = tid; r <= en; r += nthr) {
            lz v = dg[r];
            v.re -= s.re;
            v.im -= s.im;
            dg[r] = v;
            H[(long long)r * n + r] = v;
        }
        __syncthreads();

        // left half: blocks of 32 columns
        const int nblk = (en - l + 32) / 32, nout = (n - 1 - en + 31) / 32;  // blocks of the window, groups right of it
        for (int b = 0; b < nblk; ++b) {
            const int c0 = l + 32 * b;
            if (warp == 0) {
                const int nc = min(32, en - c0 + 1), cnt = min(32, en - c0);
                // the lane's entry in row c0 with the earlier blocks' rotations applied
                lz y{0, 0};
                if (b > 0) y = fix_left_block(n, H, tile, rots, c0 - 32, 32, c0, nc);
                else if (lane < nc) y = H[(long long)(c0 + lane) * n + c0];
                // the block's own rows c0 + 1 .. c0 + cnt (the upper triangle and the subdiagonal), and its
                // rotations c0 + 1 .. c0 + cnt; row c0 + i at element i
                for (int c = 1; c < nc; ++c)
                    if (lane >= 1 && lane <= c) fix_copy16(tile + c * kFixTilePitch + lane, H + (long long)(c0 + c) * n + c0 + lane);
                lz* tl = tile + lane * kFixTilePitch;
                if (lane < cnt) tl[lane + 1] = lz{sub[c0 + lane + 1], 0};
                fix_copy_wait();
                __syncwarp();
                for (int i = 1; i <= cnt; ++i) {
                    const long long xr = __shfl_sync(0xffffffffu, y.re, i - 1), xi = __shfl_sync(0xffffffffu, y.im, i - 1);
                    const lz z = tl[i];
                    const FixRot q = fix_rotation(xr, xi, sub[c0 + i]);
                    if (lane == 0) fix_put(rots + kFixEntry * (c0 + i), q);
                    lz oa, ob;
                    fix_pair<false>(q, y, z, oa, ob);
                    if (lane == i - 1) oa.im = 0;
                    if (lane >= i - 1 && lane < nc) {
                        tl[i - 1] = oa;
                        y = ob;
                    }
                }
                if (c0 + 32 > en && lane == nc - 1) {  // h(en, en): made real by a phase on column en
                    const FixRot ph = fix_rotation(y.re, y.im, 0);
                    const int has = y.im != 0;
                    if (has) {
                        const lz v = fix_phase<false>(ph, y);
                        y = lz{v.re, 0};
                    }
                    flags[48] = has;
                    fix_put(phase, ph);
                }
                if (lane < nc && lane >= cnt) tl[cnt] = y;
                __syncwarp();
                for (int c = 0; c < nc; ++c)
                    if (lane <= c) H[(long long)(c0 + c) * n + c0 + lane] = tile[c * kFixTilePitch + lane];
            } else if (b > 0) {
                // the window's columns right of this block, then the columns right of the window
                for (int g = b + warp; g < nblk + nout; g += nw - 1) {
                    const int g0 = g < nblk ? l + 32 * g : en + 1 + 32 * (g - nblk);
                    const int gc = min(32, (g < nblk ? en + 1 : n) - g0);
                    const lz y = fix_left_block(n, H, tile, rots, c0 - 32, 32, g0, gc);
                    if (lane < gc) H[(long long)(g0 + lane) * n + c0] = y;
                }
            }
            __syncthreads();
        }
        // the last block's rotations (and the phase) on the columns right of the window; the right half does not
        // touch those, so the warps with the fewest of its rows start with them
        const int has = flags[48];
        const FixRot ph = fix_get(phase);
        {
            const int r0 = l + 32 * (nblk - 1), cnt = en - r0;
            if (cnt > 0 || has)
                for (int g = nw - 1 - warp; g < nout; g += nw) {
                    const int g0 = en + 1 + 32 * g, gc = min(32, n - g0);
                    lz y{0, 0};
                    if (cnt > 0) y = fix_left_block(n, H, tile, rots, r0, cnt, g0, gc);
                    else if (lane < gc) y = H[(long long)(g0 + lane) * n + en];
                    if (has) y = fix_phase<false>(ph, y);
                    if (lane < gc) H[(long long)(g0 + lane) * n + en] = y;
                }
        }
        // right half: a lane per row, the rows above the window included; a warp's lanes go through the columns
        // together, from its first row's diagonal
        for (int r = tid; r - lane <= en; r += nthr) {
            const int r0 = r - lane, first = max(l + 1, r0);
            const bool live = r <= en;
            lz* hr = H + min(r, en);
            lz buf[kFixBatch], nxt[kFixBatch];
            lz y = live && r <= l ? hr[(long long)l * n] : zero;
            int j = first;
#pragma unroll
            for (int u = 0; u < kFixBatch; ++u) buf[u] = hr[(long long)min(j + u, en) * n];
            // up to column r0 + 32 the rows' own diagonals are met: entries left of them count as zero
            for (; j <= en && j <= r0 + 32; j += kFixBatch) {
#pragma unroll
                for (int u = 0; u < kFixBatch; ++u) nxt[u] = hr[(long long)min(j + kFixBatch + u, en) * n];
#pragma unroll
                for (int u = 0; u < kFixBatch; ++u) {
                    const int c = j + u;
                    if (c <= en) {
                        lz oa, ob;
                        fix_pair<true>(fix_get(rots + kFixEntry * c), y, c >= r ? buf[u] : zero, oa, ob);
                        y = ob;
                        if (live && c == r) sub[r] = oa.re;
                        if (live && c > r) {
                            hr[(long long)(c - 1) * n] = oa;
                            if (c == r + 1) dg[r] = oa;
                        }
                    }
                }
#pragma unroll
                for (int u = 0; u < kFixBatch; ++u) buf[u] = nxt[u];
            }
            for (; j <= en; j += kFixBatch) {
#pragma unroll
                for (int u = 0; u < kFixBatch; ++u) nxt[u] = hr[(long long)min(j + kFixBatch + u, en) * n];
#pragma unroll
                for (int u = 0; u < kFixBatch; ++u)
                    if (j + u <= en) {
                        lz oa, ob;
                        fix_pair<true>(fix_get(rots + kFixEntry * (j + u)), y, buf[u], oa, ob);
                        if (live) hr[(long long)(j + u - 1) * n] = oa;
                        y = ob;
                    }
#pragma unroll
                for (int u = 0; u < kFixBatch; ++u) buf[u] = nxt[u];
            }
            if (live) {
                if (has) y = fix_phase<true>(ph, y);
                hr[(long long)en * n] = y;
                if (r == en) dg[r] = y;
            }
        }
        for (int i = tid; i < 2 * (en - l + has); i += nthr) {
            const int k = i >> 1;  // rotation l + 1 + k, then the phase
            log[2 * pos + i] = (k < en - l ? rots + kFixEntry * (l + 1 + k) : phase)[i & 1];
        }
        if (tid == 0) table[sweeps] = make_int4(l, en, has, 0);
        pos += en - l + has;
        ++sweeps;
        __syncthreads();
    }
    if (tid == 0) {
        head[2 * gid] = sweeps;
        head[2 * gid + 1] = e2;
        status[gid] = fail;
        done[gid] = !fail;
        if (!fail) info[gid] = 0;
    }
}

// Z from the log: a lane per row, R rows (and lanes) a CTA, the row in shared memory (row t of the CTA at element
// i * R + t). A similarity H <- G H G^H takes Z <- Z G^H: (a', b') = (q a + s b, conj(q) b - s a).
template <int R = 32>
__global__ void __launch_bounds__(R) fix_apply_kernel(int n, int batch, zc* __restrict__ z_out, long long z_stride,
                                                              const int4* __restrict__ log_all, long long log_stride,
                                                              const int4* __restrict__ table_all, const int* __restrict__ head, const int* __restrict__ status) {
    RCWA_DYN_SMEM(lz, fixz_sm);
    const long long gid = blockIdx.x;
    const int lane = threadIdx.x, row = blockIdx.y * R + lane;
    if (gid >= batch || status[gid]) return;
    lz* y = fixz_sm + lane;
    for (int i = 0; i < n; ++i) y[i * R] = lz{i == row ? 1LL << 60 : 0, 0};
    // the log through shared memory: chunk c (32 rotations) in stage[c & 1], the next in registers on its way.
    // Runs of rotations are cut at the chunks' ends, so that nothing inside a run depends on the staging.
    __shared__ int4 stage[2][68];  // a run reads one rotation past its end
    const int4* log = log_all + gid * log_stride + lane;
    const int4* table = table_all + gid * fix_table_capacity(n);
    constexpr int kLoads = 64 / R;  // of a chunk's int4s, a lane
    int4 nx[kLoads];
#pragma unroll
    for (int u = 0; u < kLoads; ++u) {
        stage[0][lane + u * R] = log[u * R];
        nx[u] = log[64 + u * R];
    }
    log += 128;
    const int4* e = stage[0];
    int left = 32, b = 0;  // rotations left in the chunk
    __syncwarp();
    const auto refill = [&] {
        b ^= 1;
#pragma unroll
        for (int u = 0; u < kLoads; ++u) {
            stage[b][lane + u * R] = nx[u];
            nx[u] = log[u * R];
        }
        log += 64;
        e = stage[b];
        left = 32;
        __syncwarp();
    };
    const auto next = [&]() -> FixRot {
        if (left == 0) refill();
        const FixRot r = fix_log_get(e[0], e[1]);
        e += 2;
        --left;
        return r;
    };
    for (int k = 0; k + 1 < n; ++k) {
        const int m = n - 1 - k, len = fix_seg_len(m), ns = (m + len - 1) / len, top_row = k + 1;
        for (int sg = 0; sg < ns; ++sg) {
            const int t0 = top_row + sg * len, t1 = min(t0 + len, n);
            lz v = fix_phase<true>(next(), y[(t1 - 1) * R]);
            lz x = y[max(t1 - 2, t0) * R];
            for (int i = t1 - 2; i >= t0; --i) {
                const lz xn = y[max(i - 1, t0) * R];
                lz oa, ob;
                fix_pair<true>(next(), x, v, oa, ob);
                y[(i + 1) * R] = ob;
                v = oa;
                x = xn;
            }
            y[t0 * R] = v;
        }
        for (int d = 1; d < ns; d *= 2)
            for (int sg = 0; sg + d < ns; sg += 2 * d) {
                lz* pa = y + (top_row + sg * len) * R;
                lz* pb = y + (top_row + (sg + d) * len) * R;
                lz oa, ob;
                fix_pair<true>(next(), *pa, *pb, oa, ob);
                *pa = oa;
                *pb = ob;
            }
    }
    const int sweeps = head[2 * gid];
    for (int k = 0; k < sweeps; ++k) {
        const int4 tb = table[k];
        lz* p = y + tb.x * R;
        lz v = p[0], z = p[R];
        for (int todo = tb.y - tb.x; todo > 0;) {
            if (left == 0) refill();
            const int run = min(todo, left);
            int4 u0 = e[0], v0 = e[1];
            for (int q = 0; q < run; q += 2) {  // two a turn, each one's coefficients and entry read a turn ahead
                const int4 u1 = e[2], v1 = e[3];
                const lz z1 = p[todo - q < 2 ? R : 2 * R];
                lz oa, ob;
                fix_pair<true>(fix_log_get(u0, v0), v, z, oa, ob);
                p[0] = oa;
                v = ob;
                z = z1;
                p += R;
                e += 2;
                if (q + 1 == run) break;
                u0 = e[2];
                v0 = e[3];
                const lz z2 = p[todo - q - 1 < 2 ? R : 2 * R];
                fix_pair<true>(fix_log_get(u1, v1), v, z, oa, ob);
                p[0] = oa;
                v = ob;
                z = z2;
                p += R;
                e += 2;
            }
            todo -= run;
            left -= run;
        }
        if (tb.z) v = fix_phase<true>(next(), v);
        p[0] = v;
    }
    if (row >= n) return;
    zc* zo = z_out + gid * z_stride + row;
    for (int i = 0; i < n; ++i) zo[(long long)i * n] = zc{(double)y[i * R].re * 0x1p-60, (double)y[i * R].im * 0x1p-60};
}

// The Schur form from the reduced matrix h (lz): its upper triangle, the eigenvalues on the diagonal, zeros below;
// tn (zeroed before) receives the bit pattern of max |Re| + |Im| over T (ordered like the values).
static __global__ void fix_triangle_kernel(int n, int batch, const lz* __restrict__ h, long long h_stride, zc* __restrict__ t,
                                           long long t_stride, const zc* __restrict__ w, const int* __restrict__ head,
                                           const int* __restrict__ status, unsigned long long* __restrict__ tn) {
    const long long nn = (long long)n * n, idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= nn * batch) return;
    const long long b = idx / nn;
    if (status[b]) return;
    const int e = (int)(idx - b * nn), j = e / n, i = e - j * n;
    zc* p = t + b * t_stride + e;
    if (i > j) {
        *p = zc{0.0, 0.0};
        return;
    }
    const double unit = __longlong_as_double((long long)(head[2 * b + 1] + 1023) << 52);
    const lz v = h[b * h_stride + e];
    const zc z = i == j ? w[b * n + i] : zc{(double)v.re * unit, (double)v.im * unit};
    *p = z;
    atomicMax(tn + b, (unsigned long long)__double_as_longlong(abs1(z)));
}

// Eigenvectors of T by back substitution, 32 columns a CTA (a lane each), the columns in shared memory; the
// four warps share each dot product's terms. Coincident eigenvalues take the reference's floor and the
// entries its overflow control (include/stablercwa/eig_qr.hpp:886-951).
constexpr int kFixBackThreads = 128;
static __global__ void __launch_bounds__(kFixBackThreads) fix_backsub_kernel(int n, int batch, const zc* __restrict__ t_all,
                                                                           long long t_stride, const zc* __restrict__ w_all,
                                                                           const unsigned long long* __restrict__ tn_all,
                                                                           zc* __restrict__ x_all, long long x_stride,
                                                                           const int* __restrict__ status, double eps) {
    RCWA_DYN_SMEM(zc, fixb_sm);
    const long long gid = blockIdx.x;
    if (gid >= batch || status[gid]) return;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, j0 = blockIdx.y * 32, j = j0 + lane;
    const int jmax = min(j0 + 31, n - 1);
    zc* x = fixb_sm + lane;                       // x[k * 32]
    zc* part = fixb_sm + 32LL * n + lane;         // part[warp * 32]
    const zc* T = t_all + gid * t_stride;
    const zc* W = w_all + gid * n;
    const double rel = eps;
    double tiny = rel * __longlong_as_double((long long)tn_all[gid]);
    if (tiny == 0.0) tiny = 2.2250738585072014e-308;
    for (int k = warp; k < n; k += 4) x[k * 32] = zc{k == j ? 1.0 : 0.0, 0.0};
    __syncthreads();
    const zc wj = j < n ? W[j] : zc{0.0, 0.0};
    const double kQuotientMax = 1e300, kShrink = 0x1p-512;
    for (int i = jmax - 1; i >= 0; --i) {
        zc acc{0.0, 0.0};
#pragma unroll 4
        for (int k = i + 1 + warp; k <= jmax; k += 4) acc = zmac(T[(long long)k * n + i], x[k * 32], acc);
        part[warp * 32] = acc;
        __syncthreads();
        if (warp == 0 && i < j && j < n) {
            zc xi = (part[0] + part[32]) + (part[64] + part[96]);
            const zc wi = W[i];
            zc y = wj - wi;
            if (is_zero(y)) {
                y = zc{tiny, 0.0};
            } else {
                const double floor_value = rel * fmax(abs1(wj), abs1(wi));
                if (abs1(y) < floor_value) y = zc{floor_value, 0.0};
            }
            for (int pass = 0; pass < 3 && abs1(xi) > abs1(y) * kQuotientMax; ++pass) {
                xi = xi * kShrink;
                for (int k = i + 1; k <= j; ++k) x[k * 32] = x[k * 32] * kShrink;
            }
            xi = zdiv(xi, y);
            const double tr = abs1(xi);
            if (tr > 1e15 && tr + 1.0 / tr <= tr) {
                xi = zdivr(xi, tr);
                for (int k = i + 1; k <= j; ++k) x[k * 32] = zdivr(x[k * 32], tr);
            }
            x[i * 32] = xi;
        }
        __syncthreads();
    }
    for (int c = warp; c < 32 && j0 + c < n; c += 4) {
        zc* out = x_all + gid * x_stride + (long long)(j0 + c) * n;
        for (int k = lane; k < n; k += 32) out[k] = k <= j0 + c ? fixb_sm[k * 32 + c] : zc{0.0, 0.0};
    }
}

// columns of V to unit 2-norm, a warp per column (include/stablercwa/eig_qr.hpp:953-961)
static __global__ void __launch_bounds__(128) fix_unit_columns_kernel(int n, int batch, zc* __restrict__ v, long long v_stride,
                                                                      const int* __restrict__ status) {
    const long long gw = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (gw >= (long long)batch * n) return;
    const long long b = gw / n;
    if (status[b]) return;
    const int lane = threadIdx.x & 31;
    zc* c = v + b * v_stride + (gw - b * n) * n;
    double big = 0.0;
    for (int r = lane; r < n; r += 32) big = fmax(big, fmax(fabs(c[r].re), fabs(c[r].im)));
    big = group_max<32>(big, 0xffffffffu);
    if (big == 0.0 || !isfinite(big)) return;
    double ssq = 0.0;
    for (int r = lane; r < n; r += 32) ssq += norm2(zdivr(c[r], big));
    ssq = group_sum<32>(ssq, 0xffffffffu);
    const double inv = 1.0 / sqrt(ssq);
    for (int r = lane; r < n; r += 32) c[r] = zdivr(c[r], big) * inv;
}

// ---------------------------------------------------------------- the Hermitian solver's QL iteration
//
// herm_ql_kernel's iteration (eig.cuh: implicit QL with Wilkinson's shift on d and e, one thread per matrix, every
// rotation logged for herm_apply_real_kernel) in fixed point. Its chain of about 20 dependent FP64 instructions a
// rotation, 64 cycles each, took 1.1 us (17.2 ms for one matrix of order 121); the same chain in integers takes
// 0.6 us (9.2 ms), and 4096 matrices' 20 ms went to 10. d and e are scaled so that
// N >= ||T||_2 (Gershgorin's bound) lies in [2^58, 2^59) units: the iteration's quantities stay below 4 N. In memory d
// and e have three more bits (|d|, |e| <= N fit), in the chain thirty (FixWide): with whole units throughout (7.4 ms),
// the eigenvalues that are small beside N, a grating layer's propagating modes, came out up to three times as far off
// as FP64's, whose rounding follows the entries; now they are closer (reflection amplitudes of order-301 layers, mean
// relative error: FP64 5.4e-12, whole units 1.4e-11, these 2.2e-12). What it does
// not finish (non-finite or zero matrices, scales whose powers of two are not normal doubles, 30 sweeps without a
// deflation) is flagged as a full log is, for the fused FP64 kernel. status, if given: 1 for matrices whose reduction
// left them to that kernel already, kFixOther for those of herm_ql_kernel.
constexpr int kFixQlBits = 59;
constexpr int kFixQlExtra = 3;  // bits below one unit of d and e in memory

struct FixWide {  // y + x 2^-30 units, x in [0, 2^30)
    long long y;
    int x;
};
__device__ __forceinline__ FixWide fix_wide_unpack(long long v) {
    return FixWide{v >> kFixQlExtra, (int)((unsigned)v & ((1u << kFixQlExtra) - 1)) << (30 - kFixQlExtra)};
}
__device__ __forceinline__ long long fix_wide_pack(const FixWide& a) {
    return a.y * (1 << kFixQlExtra) + ((a.x + (1 << (29 - kFixQlExtra))) >> (30 - kFixQlExtra));
}
__device__ __forceinline__ FixWide fix_wide_add(const FixWide& a, const FixWide& b) {
    const int x = a.x + b.x;
    return FixWide{a.y + b.y + (x >> 30), x & 0x3fffffff};
}
__device__ __forceinline__ FixWide fix_wide_sub(const FixWide& a, const FixWide& b) {
    const int x = a.x - b.x;
    return FixWide{a.y - b.y + (x >> 30), x & 0x3fffffff};
}
// a b with the coefficient a = (a1, a0)
__device__ __forceinline__ FixWide fix_wide_mul(int a1, int a0, const FixWide& b) {
    const FixLimb l = fix_split(b.y);
    const long long u2 = fix_mad(a0, l.l, fix_mad(a1, b.x, 1LL << 29));
    const long long u = fix_mad(a0, l.h, fix_mad(a1, l.l, u2 >> 30));
    return FixWide{fix_mad(a1, l.h, u >> 30), (int)((unsigned)u & 0x3fffffffu)};
}
// a b + c d; d's terms last
__device__ __forceinline__ FixWide fix_wide_dot(int a1, int a0, const FixWide& b, int c1, int c0, const FixWide& d) {
    const FixLimb l = fix_split(b.y), m = fix_split(d.y);
    long long u2 = fix_mad(a0, l.l, fix_mad(a1, b.x, 1LL << 29));
    long long u = fix_mad(a0, l.h, fix_mad(a1, l.l, 0));
    u2 = fix_mad(c0, m.l, fix_mad(c1, d.x, u2));
    u = fix_mad(c0, m.h, fix_mad(c1, m.l, u)) + (u2 >> 30);
    return FixWide{fix_mad(c1, m.h, fix_mad(a1, l.h, 0)) + (u >> 30), (int)((unsigned)u & 0x3fffffffu)};
}
static __global__ void __launch_bounds__(kHermQlThreads) herm_ql_fixed_kernel(int n, int batch, zc* __restrict__ w,
                                                                             int* __restrict__ info, zc* __restrict__ ws,
                                                                             const int* __restrict__ status,
                                                                             unsigned long long* rotations) {
    RCWA_DYN_SMEM(long long, fixq_sm);
    const long long gid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (gid >= batch) return;
    zc* base = ws + gid * eig_workspace_elems(n);
    const double* src = reinterpret_cast<const double*>(base + 2LL * n * n);
    int* tail = reinterpret_cast<int*>(base + 3LL * n * n);  // [0] sweeps, [1] left to the fused kernel
    long long* d = fixq_sm + threadIdx.x;
    const int sd = blockDim.x;
    long long* e = d + n * sd;
    // the scale
    float big = 0.0f;
    int e2 = 0;
    const int set = status ? status[gid] : 0;
    bool usable = set == 0;
    if (usable) {
        int top = 0;
        for (int k = 0; k < 2 * n; ++k) top = max(top, (int)((__double_as_longlong(src[k]) >> 52) & 0x7FF));
        usable = top >= 200 && top <= 1900;
        if (usable) {
            const double scl = __longlong_as_double((long long)(2046 - top) << 52);
            float below = 0.0f;
            for (int k = 0; k < n; ++k) {
                const float ek = k + 1 < n ? fabsf((float)(src[n + k] * scl)) : 0.0f;
                big = fmaxf(big, fabsf((float)(src[k] * scl)) + ek + below);
                below = ek;
            }
            e2 = ((__float_as_int(big * 1.001f) >> 23) & 0xff) - 127 + 1 + (top - 1023) - kFixQlBits;
        }
    }
    if (set != kFixOther) {
        tail[0] = 0;
        tail[1] = !usable;
        info[gid] = 0;
    }
    if (!usable) return;
    for (int k = 0; k < n; ++k) {
        d[k * sd] = fix_from_double(src[k], e2 - kFixQlExtra);
        e[k * sd] = k + 1 < n ? fix_from_double(src[n + k], e2 - kFixQlExtra) : 0;
    }
    int2* table = reinterpret_cast<int2*>(reinterpret_cast<double*>(base) + 2 * n);
    int4* log = reinterpret_cast<int4*>(base + (long long)n * n);
    const long long log_cap = herm_log_capacity(n), table_cap = herm_table_capacity(n);
    long long pos = 0, sweeps = 0;
    bool left = false;
    for (int l = 0; l < n && !left; ++l) {
        for (int its = 0;; ++its) {
            // first m >= l with e[m] below eps (|d[m]| + |d[m+1]|), or of half a unit (2^-59 N at most)
            int m = l;
            for (; m < n - 1; ++m) {
                const long long a = d[m * sd], b = d[(m + 1) * sd], x = e[m * sd];
                const unsigned long long size = (unsigned long long)((a < 0 ? -a : a) + (b < 0 ? -b : b));
                const unsigned long long ax = (unsigned long long)(x < 0 ? -x : x);
                if (ax <= 4 || ax <= size >> 52) break;
            }
            if (m == l) break;
            if (its == 30 || pos + (m - l) > log_cap || sweeps + 1 > table_cap) {
                left = true;
                break;
            }
            // g = d[m] - shift, the shift d[l] - e^2 / (h + sign(h) sqrt(h^2 + e^2)), h = (d[l+1] - d[l]) / 2, its
            // correction in float
            FixWide g = fix_wide_sub(fix_wide_unpack(d[m * sd]), fix_wide_unpack(d[l * sd]));
            {
                const float k = 0x1p-62f;  // 2^-59 units
                const float h = (float)((d[(l + 1) * sd] >> 1) - (d[l * sd] >> 1)) * k, x = (float)e[l * sd] * k;
                const float den = h + copysignf(sqrtf(h * h + x * x), h);
                if (fabsf(den) > 1e-18f) g.y += (long long)(x * (x / den) * 0x1p59f);
            }
            FixRot q;  // c and s of the last rotation (c in q.cr, s in q.s)
            q.cr1 = q.s1 = 1 << 30;
            q.cr0 = q.s0 = 0;
            FixWide p{0, 0};
            bool split = false;
            int i = m - 1;
            FixWide ei = fix_wide_unpack(e[i * sd]), di = fix_wide_unpack(d[i * sd]), dn = fix_wide_unpack(d[m * sd]);
            for (; i >= l; --i) {
                const FixLimb el = fix_split(ei.y);
                const FixWide b = fix_wide_mul(q.cr1, q.cr0, ei);
                // f = s e to the last digit, 60 fractional bits in fl: where f and g are both small the angle between
                // them, which carries the shift up the matrix, needs f's digits below one unit
                const long long ll = fix_mad(q.s0, el.l, fix_mad(q.s1, ei.x, fix_mad(q.s0, ei.x, 0) >> 30)),
                                u = fix_mad(q.s0, el.h, fix_mad(q.s1, el.l, ll >> 30));
                const FixWide f{fix_mad(q.s1, el.h, u >> 30), (int)((unsigned)u & 0x3fffffffu)};
                const unsigned long long fl = (unsigned long long)f.x << 30 | ((unsigned)ll & 0x3fffffffu);
                // the next rotation's entries, ahead of their use
                const int in = i > l ? i - 1 : l;
                const long long en = e[in * sd], dp = d[in * sd];
                if (f.y == 0 && fl == 0 && g.y == 0 && g.x == 0) {
                    e[(i + 1) * sd] = 0;
                    d[(i + 1) * sd] = fix_wide_pack(fix_wide_sub(dn, p));
                    e[m * sd] = 0;
                    split = true;
                    break;
                }
                {
                    long long x = g.y, y = f.y;
                    unsigned long long r = fl, rx = (unsigned long long)g.x << 30;
                    int h = fix_tops(x, y, 0);
                    while (h == 0) {
                        x = (long long)((unsigned long long)x << 28 | rx >> 32);
                        rx = (rx << 28) & 0xfffffffffffffffull;
                        y = (long long)((unsigned long long)y << 28 | r >> 32);
                        r = (r << 28) & 0xfffffffffffffffull;
                        h = fix_tops(x, y, 0);
                    }
                    const int sh = __clz(h) - 3;
                    q = fix_rotation_scaled((long long)((unsigned long long)x << sh | rx >> (60 - sh)), 0,
                                            (long long)((unsigned long long)y << sh | r >> (60 - sh)));
                }
                e[(i + 1) * sd] = fix_wide_pack(fix_wide_dot(q.s1, q.s0, f, q.cr1, q.cr0, g));
                const FixWide g2 = fix_wide_sub(dn, p);
                const FixWide t = fix_wide_dot(q.cr1, q.cr0, fix_wide_add(b, b), q.s1, q.s0, fix_wide_sub(di, g2));
                p = fix_wide_mul(q.s1, q.s0, t);
                d[(i + 1) * sd] = fix_wide_pack(fix_wide_add(g2, p));
                g = fix_wide_sub(fix_wide_mul(q.cr1, q.cr0, t), b);
                // the log's form (herm_fixed_entry): s 2^62 and -c 2^62 in 31-bit limbs, saturated below 2^62
                const long long s62 = min((((long long)q.s1 << 30) + q.s0) << 2, 0x3fffffffffffffffLL),
                                c62 = min((((long long)q.cr1 << 30) + q.cr0) << 2, 0x3fffffffffffffffLL);
                const long long S = max(s62, -0x3fffffffffffffffLL), C = -max(c62, -0x3fffffffffffffffLL);
                log[pos] = make_int4((int)(S >> 31), (int)(S & 0x7fffffff), (int)(C >> 31), (int)(C & 0x7fffffff));
                ++pos;
                dn = di;
                ei = fix_wide_unpack(en);
                di = fix_wide_unpack(dp);
            }
            const int first = split ? i + 1 : l;
            if (!split) {
                d[l * sd] = fix_wide_pack(fix_wide_sub(dn, p));
                e[l * sd] = fix_wide_pack(g);
                e[m * sd] = 0;
            }
            if (m - 1 >= first) table[sweeps++] = make_int2(first, m - 1);
        }
    }
    tail[0] = (int)sweeps;
    tail[1] = left;
    if (!left) {
        const double unit = __longlong_as_double((long long)(e2 - kFixQlExtra + 1023) << 52);
        for (int k = 0; k < n; ++k) w[gid * n + k] = zc{(double)d[k * sd] * unit, 0.0};
        if (rotations) atomicAdd(rotations, (unsigned long long)pos);
    }
}

}  // namespace rcwa_gb300
