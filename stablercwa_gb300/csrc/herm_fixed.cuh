// herm_fixed.cuh -- the panels of the blocked Hermitian tridiagonalisation (eig.cuh herm_panel_one) with their
// matrix-vector products in 64-bit fixed point.
//
// The panel's FP64 work is the product with the trailing block and six passes over the earlier reflectors a
// column; at 64 cycles a warp instruction it kept the FP64 pipe 79 % busy (66.5 ms for 4096 matrices of order
// 121). The same sums run on the integer pipes, 12 multiply-adds of 2 cycles a complex term instead of 4 of 64:
// 37.9 ms, of which the reads of the trailing block would take 13 at the memory's rate and the FP64 that is left (a
// column's scalars, T and M = T V^H) about 10. What bounds it is latency at 6.8 warps an SM: waits for the trailing
// block's entries, the integer pipes 12 to 20 % and the FP64 pipe 18 to 45 % busy (1024 matrices).
//
// The matrix is scaled once by a power of two, which d and e undo, so that N, its largest row sum of |re| + |im|
// (>= ||A||_2), is below 1. A panel holds its trailing block in units of 2^-(60 + s), s <= 2 as its largest entry
// allows (y = A v stays below 2^63), the reflectors (|v_r| <= 1, ||v||^2 <= 2) with 59 fractional bits, each w in
// units of 2^-60 of its own norm's power of two. Each component is a pair of limbs h 2^30 + l with l in
// [-2^29, 2^29), two components an int4, the size of the complex double. A product keeps
// h h' and (h l' + l h') 2^-30; l l' (zero mean, a sixth of a unit rms) is dropped. The sums of h h' may wrap: the
// result fits. y is then off by about 4 units, 2^-58 N to 2^-60 N; FP64 rounds y's entries (of the size N / sqrt(n))
// at 2^-53 of themselves, every partial sum again. The scalars of a column, v, w and T stay in FP64.
#pragma once

#include <climits>

#include "eig_fixed.cuh"

namespace rcwa_gb300 {

constexpr int kHermFixV = 59;  // fractional bits of the reflectors
constexpr long long kHermFixHalf = 1LL << (kHermFixV - 31);

// a running complex sum: high products, middle products (flushed before they pass 2^63, rounded), flushed part
struct HermFixSum {
    long long hr, mr, fr, hi, mi, fi;
    __device__ __forceinline__ HermFixSum() : hr(0), mr(kHermFixHalf), fr(0), hi(0), mi(kHermFixHalf), fi(0) {}
    __device__ __forceinline__ void flush() {
        fr += mr >> (kHermFixV - 30);
        fi += mi >> (kHermFixV - 30);
        mr = mi = kHermFixHalf;
    }
    __device__ __forceinline__ long long re() const { return 2 * hr + fr; }
    __device__ __forceinline__ long long im() const { return 2 * hi + fi; }
};
// y's limbs (real h, l, imaginary h, l) with the imaginary part's negatives beside them
struct HermFixCoef {
    int rh, rl, ih, il, nh, nl;
};
__device__ __forceinline__ HermFixCoef herm_fix_coef(const int4& y) { return HermFixCoef{y.x, y.y, y.z, y.w, -y.z, -y.w}; }
__device__ __forceinline__ HermFixCoef herm_fix_conj(const int4& y) { return HermFixCoef{y.x, y.y, -y.z, -y.w, y.z, y.w}; }
__device__ __forceinline__ HermFixCoef herm_fix_neg(const int4& y) { return HermFixCoef{-y.x, -y.y, -y.z, -y.w, y.z, y.w}; }
__device__ __forceinline__ HermFixCoef herm_fix_neg_conj(const int4& y) { return HermFixCoef{-y.x, -y.y, y.z, y.w, -y.z, -y.w}; }
// s += x y
__device__ __forceinline__ void herm_fix_mac(HermFixSum& s, const int4& x, const HermFixCoef& y) {
    s.hr = fix_mad(x.x, y.rh, s.hr);
    s.hi = fix_mad(x.x, y.ih, s.hi);
    s.mr = fix_mad(x.x, y.rl, s.mr);
    s.mi = fix_mad(x.x, y.il, s.mi);
    s.hr = fix_mad(x.z, y.nh, s.hr);
    s.hi = fix_mad(x.z, y.rh, s.hi);
    s.mr = fix_mad(x.y, y.rh, s.mr);
    s.mi = fix_mad(x.y, y.ih, s.mi);
    s.mr = fix_mad(x.z, y.nl, s.mr);
    s.mi = fix_mad(x.z, y.rl, s.mi);
    s.mr = fix_mad(x.w, y.nh, s.mr);
    s.mi = fix_mad(x.w, y.rh, s.mi);
}
__device__ __forceinline__ int4 herm_fix_limbs(long long re, long long im) {
    int4 v;
    fix_limbs(re, v.x, v.y);
    fix_limbs(im, v.z, v.w);
    return v;
}
__device__ __forceinline__ int4 herm_fix_limbs(const zc& z, int e) {
    return herm_fix_limbs(fix_from_double(z.re, e), fix_from_double(z.im, e));
}
__device__ __forceinline__ long long herm_fix_join(int h, int l) { return (long long)h * (1LL << 30) + l; }
// x 2^t, rounded
__device__ __forceinline__ long long herm_fix_shift(long long x, int t) {
    return t >= 0 ? (long long)((unsigned long long)x << t) : (x + (1LL << (-t - 1))) >> -t;
}
__device__ __forceinline__ double herm_fix_pow2(int e) { return __longlong_as_double((long long)(e + 1023) << 52); }
template <int G>
__device__ __forceinline__ long long herm_fix_group_sum(long long v, unsigned mask) {
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) v += __shfl_xor_sync(mask, v, o, G);
    return v;
}

// rows i0 + u G (u < U) of y = A v over columns c0 .. n - 1
template <int G, int U>
__device__ __forceinline__ void herm_fix_rows(int n, int c0, int i0, const int4* __restrict__ LA, const int4* __restrict__ v,
                                              lz* __restrict__ y) {
    HermFixSum s[U];
    const int4* a[U];
#pragma unroll
    for (int u = 0; u < U; ++u) a[u] = LA + min(i0 + u * G, n - 1);
    for (int c = c0; c < n; c += 2) {
        const int c1 = min(c + 1, n - 1);
        int4 v1 = v[c1];
        if (c1 == c) v1 = make_int4(0, 0, 0, 0);
        const HermFixCoef x0 = herm_fix_coef(v[c]), x1 = herm_fix_coef(v1);
        int4 a0[U], a1[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            a0[u] = a[u][(long long)c * n];
            a1[u] = a[u][(long long)c1 * n];
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            herm_fix_mac(s[u], a0[u], x0);  // middle terms below 2^60.6 a product
            herm_fix_mac(s[u], a1[u], x1);
            s[u].flush();
        }
    }
#pragma unroll
    for (int u = 0; u < U; ++u)
        if (i0 + u * G < n) y[i0 + u * G] = lz{s[u].re(), s[u].im()};
}

// herm_panel_one with the sums in fixed point; 2^ex: the scale taken out of A.
template <int G>
__device__ void herm_panel_fixed(int n, int k0, int ex, zc* __restrict__ ws, zc* __restrict__ pan, zc* __restrict__ vall,
                                 zc* __restrict__ mall, int pnb) {
    constexpr int nb = kHermNb;
    const int g = threadIdx.x & (G - 1);
    const Grp<G> grp(nullptr, nullptr);
    zc* A = ws;
    int4* LA = reinterpret_cast<int4*>(ws + (long long)n * n);  // A's limbs
    double* __restrict__ d = reinterpret_cast<double*>(ws + 2LL * n * n);
    double* __restrict__ e = d + n;
    zc* ww = ws + 3LL * n * n;
    lz* yy = reinterpret_cast<lz*>(ww);  // y in units, then in FP64 in the same place
    zc* __restrict__ taus = ww + n;
    zc* __restrict__ VW = pan;
    zc* Bt = pan + 2LL * nb * n;
    int4* LV = reinterpret_cast<int4*>(Bt);  // V's and W's limbs, in Bt's place until it is written
    int4* LW = LV + (long long)nb * n;
    zc* __restrict__ T = Bt + 2LL * nb * n;
    zc* t2 = T + nb * nb;
    lz* t2raw = reinterpret_cast<lz*>(t2);
    const int nbp = min(nb, n - 1 - k0);
    int* wex = reinterpret_cast<int*>(ws + 3LL * n * n + 2 * n) + 1;  // the exponents of the w's norms
    int top = 0;
    for (int c = k0; c < n; ++c)
        for (int r = first_owned<G>(k0, g); r < n; r += G) {
            const zc z = A[(long long)c * n + r];
            top = max(top, max((int)(__double_as_longlong(z.re) >> 52 & 0x7FF), (int)(__double_as_longlong(z.im) >> 52 & 0x7FF)));
        }
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) top = max(top, __shfl_xor_sync(grp.mask, top, o, G));
    const int s_a = min(2, max(0, 1022 - top)), ea = -60 - s_a;  // |entries| < 2^-s_a
    const double unit = herm_fix_pow2(ea), back = herm_fix_pow2(ex);
    const zc one{1.0, 0.0}, zero{0.0, 0.0};
    const int4 lzero = make_int4(0, 0, 0, 0);
    for (int c = k0; c < n; ++c)
        for (int r = first_owned<G>(k0, g); r < n; r += G) LA[(long long)c * n + r] = herm_fix_limbs(A[(long long)c * n + r], ea);
    for (int c = 0; c < 2 * nb; ++c)
        for (int r = g; r < n; r += G) {
            VW[(long long)c * n + r] = zero;
            LV[(long long)c * n + r] = lzero;
        }
    for (int idx = g; idx < nb * nb; idx += G) T[idx] = zero;
    grp.sync();
    for (int i = 0; i < nbp; ++i) {
        const int j = k0 + i;
        zc* col = A + (long long)j * n;
        const int4* lv = LV + (long long)i * n;
        // column j as the panel's earlier reflectors leave it (rows >= j)
        for (int r = first_owned<G>(j, g); r < n; r += G) {
            const int4 a = LA[(long long)j * n + r];
            lz v{herm_fix_join(a.x, a.y), herm_fix_join(a.z, a.w)};
#pragma unroll 2
            for (int p = 0; p < i; ++p) {
                HermFixSum s;
                herm_fix_mac(s, LV[(long long)p * n + r], herm_fix_neg_conj(LW[(long long)p * n + j]));
                herm_fix_mac(s, LW[(long long)p * n + r], herm_fix_neg_conj(LV[(long long)p * n + j]));
                s.flush();
                const int t = wex[p] + s_a;
                v.re += herm_fix_shift(s.re(), t);
                v.im += herm_fix_shift(s.im(), t);
            }
            col[r] = zc{(double)v.re * unit, (double)v.im * unit};
        }
        grp.sync();
        if (g == 0) d[j] = col[j].re * back;
        const zc alpha = col[j + 1];
        const int r2 = first_owned<G>(j + 2, g), r1 = first_owned<G>(j + 1, g);
        double xs = 0.0;
        for (int r = r2; r < n; r += G) xs += norm2(col[r]);
        xs = grp.sum(xs);
        zc tau{0.0, 0.0};
        double beta = alpha.re;
        zc scal = zero;
        if (xs != 0.0 || alpha.im != 0.0) {
            const double nrm = hypot(hypot(alpha.re, alpha.im), sqrt(xs));
            beta = alpha.re >= 0.0 ? -nrm : nrm;
            tau = zc{(beta - alpha.re) / beta, -alpha.im / beta};
            scal = zinv(alpha - zc{beta, 0.0});
        }
        if (g == 0) {
            e[j] = beta * back;
            taus[j] = tau;
        }
        zc* __restrict__ vcol = vall + (long long)j * n;
        for (int r = g; r < n; r += G) {
            const zc vr = r <= j ? zero : (r == j + 1 ? one : col[r] * scal);
            vcol[r] = vr;
            VW[(long long)i * n + r] = vr;
            if (r > j) LV[(long long)i * n + r] = herm_fix_limbs(vr, -kHermFixV);
        }
        grp.sync();  // v is complete
        if (is_zero(tau)) {  // H_j = I: w = 0 and T's column is zero (both already)
            if (g == 0) wex[i] = 0;
            grp.sync();  // the next column's updates read it
            continue;
        }
        // y = A0 v over the trailing block, owned rows, up to four a pass
        int i0 = r1;
        for (; i0 + 3 * G < n + G; i0 += 4 * G) herm_fix_rows<G, 4>(n, j + 1, i0, LA, lv, yy);
        for (; i0 < n; i0 += G) herm_fix_rows<G, 1>(n, j + 1, i0, LA, lv, yy);
        // y -= V (W^H v) + W (V^H v), one earlier reflector at a time
        for (int p = 0; p < i; ++p) {
            const int4* vp = LV + (long long)p * n;
            const int4* wp = LW + (long long)p * n;
            HermFixSum a1, a2;
#pragma unroll 2
            for (int r = r1; r < n; r += G) {
                const int4 vr = lv[r];
                herm_fix_mac(a1, vr, herm_fix_conj(wp[r]));
                herm_fix_mac(a2, vr, herm_fix_conj(vp[r]));
                a1.flush();
                a2.flush();
            }
            const long long s1r = herm_fix_group_sum<G>(a1.re(), grp.mask), s1i = herm_fix_group_sum<G>(a1.im(), grp.mask);
            const long long s2r = herm_fix_group_sum<G>(a2.re(), grp.mask), s2i = herm_fix_group_sum<G>(a2.im(), grp.mask);
            const int t = wex[p] + s_a;
            const HermFixCoef c1 = herm_fix_neg(herm_fix_limbs(s1r, s1i)), c2 = herm_fix_neg(herm_fix_limbs(s2r, s2i));
#pragma unroll 2
            for (int r = r1; r < n; r += G) {
                HermFixSum s;
                herm_fix_mac(s, vp[r], c1);
                herm_fix_mac(s, wp[r], c2);
                s.flush();
                const lz y = yy[r];
                yy[r] = lz{y.re + herm_fix_shift(s.re(), t), y.im + herm_fix_shift(s.im(), t)};
            }
            if (g == 0) t2raw[p] = lz{s2r, s2i};
        }
        const zc* __restrict__ v64 = VW + (long long)i * n;
        double mr = 0.0;
        for (int r = r1; r < n; r += G) {
            const lz y = yy[r];
            const zc w{(double)y.re * unit, (double)y.im * unit}, vr = v64[r];
            ww[r] = w;
            mr += vr.re * w.re + vr.im * w.im;  // Re(conj(v_r) y_r)
        }
        const double half = 0.5 * norm2(tau) * grp.sum(mr);
        double wn = 0.0;
        zc* wi = VW + (long long)(nb + i) * n;
        for (int r = r1; r < n; r += G) {
            const zc vr = v64[r];
            const zc w = tau * ww[r] - zc{half * vr.re, half * vr.im};
            wi[r] = w;
            wn += norm2(w);
        }
        wn = grp.sum(wn);
        // ||w|| < 2^xw, 2^-61 <= 2^xw <= 4 (a smaller w is below every unit)
        const int xw = min(2, max(-61, (((int)(__double_as_longlong(wn) >> 52) & 0x7FF) - 1021) >> 1));
        if (g == 0) wex[i] = xw;
        for (int r = r1; r < n; r += G) LW[(long long)i * n + r] = herm_fix_limbs(wi[r], xw - 60);
        grp.sync();  // t2 is complete
        for (int p = g; p < i; p += G) {
            const lz s = t2raw[p];
            const double f = herm_fix_pow2(-kHermFixV);
            t2[p] = zc{(double)s.re * f, (double)s.im * f};
        }
        grp.sync();
        // T(0:i, i) = -tau T(0:i, 0:i) t2, T(i, i) = tau
        for (int p = g; p < i; p += G) {
            zc z = zero;
            for (int q = p; q < i; ++q) z = zmac(T[q * nb + p], t2[q], z);
            T[i * nb + p] = zc{0.0, 0.0} - tau * z;
        }
        if (g == 0) T[i * nb + i] = tau;
        grp.sync();  // w and T's column are complete
    }
    if (k0 + nbp == n - 1 && g == 0) {  // the last panel: the last diagonal entry takes its updates too
        zc a = A[(long long)(n - 1) * n + n - 1];
        for (int p = 0; p < nbp; ++p) {
            a = zfms(VW[(long long)p * n + n - 1], conj(VW[(long long)(nb + p) * n + n - 1]), a);
            a = zfms(VW[(long long)(nb + p) * n + n - 1], conj(VW[(long long)p * n + n - 1]), a);
        }
        d[n - 1] = a.re * back;
        e[n - 1] = 0.0;
    }
    herm_panel_finish<G>(n, k0, nbp, VW, Bt, T, mall, pnb);
}

// The scale of the Hermitian part: 2^ex > N, or INT_MIN where N is zero, not finite or far from 1 (the FP64
// panels take the matrix, as they do where other[b] is set).
template <int G>
__device__ int herm_fix_scale(int n, const zc* __restrict__ A0) {
    const int g = threadIdx.x & (G - 1);
    const Grp<G> grp(nullptr, nullptr);
    double top = 0.0, bad = 0.0;
    for (int r = g; r < n; r += G) {
        double sum = 0.0;
        for (int c = 0; c < n; ++c) {
            const zc a = A0[(long long)c * n + r], b = A0[(long long)r * n + c];
            const zc h{0.5 * (a.re + b.re), 0.5 * (a.im - b.im)};
            sum += fabs(h.re) + fabs(h.im);
        }
        if (!(sum < 1e290)) bad = 1.0;
        top = fmax(top, sum);
    }
    top = grp.max(top);
    bad = grp.sum(bad);
    if (bad != 0.0 || !(top > 1e-290)) return INT_MIN;
    return (int)((__double_as_longlong(top) >> 52) & 0x7FF) - 1022;
}

template <int G>
__global__ void __launch_bounds__(128) herm_panel_fixed_kernel(int n, int batch, int k0, const zc* __restrict__ a, long long a_stride,
                                                               zc* __restrict__ ws, zc* __restrict__ pan, zc* __restrict__ vall,
                                                               zc* __restrict__ mall, int pnb, const int* __restrict__ other = nullptr) {
    const long long gid = ((long long)blockIdx.x * blockDim.x + threadIdx.x) / G;
    if (gid >= batch) return;
    zc* w = ws + gid * eig_workspace_elems(n);
    zc* p = pan + gid * herm_panel_elems(n);
    zc* va = vall + gid * (long long)n * n;
    zc* ma = mall + gid * (long long)pnb * n;
    const zc* A0 = a + gid * a_stride;
    int* head = reinterpret_cast<int*>(w + 3LL * n * n + 2 * n);
    int ex;
    if (k0 == 0) {
        const int g = threadIdx.x & (G - 1);
        const Grp<G> grp(nullptr, nullptr);
        ex = other && other[gid] ? INT_MIN : herm_fix_scale<G>(n, A0);
        if (g == 0) *head = ex;
        if (ex != INT_MIN) {
            const double half = herm_fix_pow2(-ex - 1);
            for (int c = 0; c < n; ++c)
                for (int r = g; r < n; r += G) {
                    const zc x = A0[(long long)c * n + r], y = A0[(long long)r * n + c];
                    w[(long long)c * n + r] = zc{half * (x.re + y.re), half * (x.im - y.im)};
                }
            grp.sync();
        }
    } else {
        ex = *head;
    }
    if (ex == INT_MIN) herm_panel_one<G>(n, k0, A0, w, p, va, ma, pnb);
    else herm_panel_fixed<G>(n, k0, ex, w, p, va, ma, pnb);
}

}  // namespace rcwa_gb300
