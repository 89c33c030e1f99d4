// gemm_tc.cu -- batched complex FP64 GEMM on the tensor cores (tcgen05, sm_103a), accurate to FP64.
//
// C = s_ab A B + s_c C0 with A m x k, B k x n complex double, any batch. The product is emulated with
// the Ozaki scheme (Ozaki, Ogita, Oishi and Rump, "Error-free transformations of matrix
// multiplication by using fast routines of matrix multiplication", Numer. Algorithms 59, 2012) on
// bf16 tensor-core products:
//   * the complex product is one real product of twice the size: rows 2i and 2i+1 of A^ are
//     [Re A(i,:), -Im A(i,:)] and [Im A(i,:), Re A(i,:)], and B^ = [Re B; Im B], so (A^ B^)(2i, j) and
//     (A^ B^)(2i+1, j) are the real and imaginary parts of C(i, j);
//   * every row of A^ is scaled by a power of two 2^ea(i) taken from its largest entry, every column of
//     B^ by 2^eb(j), and each scaled entry y in (-1, 1) is split into S signed integer digits,
//     y = 2^-7 (d_1 + 2^-8 d_2 + ... + 2^-8(S-1) d_S), |d_s| <= 128: each digit is exact in bf16;
//   * the digit products d_s e_t are exact (<= 2^14) and a tensor-core sum of up to 1024 of them stays
//     an integer below 2^24, exact in the FP32 accumulator. Digit pairs (s, t) with s + t <= S + 1 are
//     kept (the dropped ones lie below 2^-8S of the product's scale); pairs of one diagonal s + t share
//     a scale factor 2^(-14 - 8 (s + t - 2)), so up to 1024 / K of them accumulate in one exact FP32
//     tensor-memory accumulator (a "group") before it is added, exactly, into an int64 per element.
// Per element the result is exact up to the digit truncation (relative 2^-8S of max|A(i,:)| max|B(:,j)|
// times k) and one final rounding: FP64-level accuracy with S = 7.
//
// Kernels. The split kernels write the digit planes in HBM as bf16 rows with K contiguous (K-major for
// both operands), the second half of a complex K starting at Kp / 2. The product kernel gives each CTA one
// 128 x 128 tile of C^ of one matrix: one warp issues TMA loads (128-byte swizzle, boxes of 128 rows x 64 K, two
// of each operand a stage: two digits of 64 K, or one of 128 K) into a 3-stage shared-memory ring; one thread issues tcgen05.mma (M = 128, N = 256 or 128,
// K = 16, bf16 in, FP32 out) into four 128-column tensor-memory accumulators; eight warps read each finished
// accumulator out of tensor memory (tcgen05.ld) and add it, as an integer at its diagonal's weight, into one int64 per
// element while the next group accumulates in other slots, then convert once, apply 2^(ea + eb), pair the
// real and imaginary rows and write C. Every mbarrier wait is bounded: on expiry the kernel records an error,
// drains its own copies and products, frees its tensor memory and returns without writing C.
//
// Shared memory bounds the products: an MMA of N = 128 reads 8 KB of operands in the 64 cycles it takes, 128 bytes a
// cycle, all there is, and the copies write there too. So digits go in quads, two of A and two of B a stage: four
// digit products for four boxes instead of two, and A_i meets both of B's in one MMA of N = 256 (12 KB in 128 cycles).
// Order 121: a pair and 128 K a stage took 1430 cycles a stage (80,000 a tile), quads with N = 128 MMAs 1575 (68,000, at
// 125 bytes a cycle); 4096 products with their digit splits 4.65, 4.39 and, with N = 256, 4.27 ms; 64 of order 301
// 0.856, 0.831, 0.766. With K = 32 (the factorisations' updates) the three are equal: loads and the conversion bound those.
#include <cuda.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <type_traits>
#include <vector>

#include "engine.h"

namespace rcwa_gb300 {
namespace {

// A stage holds two boxes of each operand (64 bf16 = one 128-byte swizzle row a box): of a quad 64 K of two digits of
// each, in eight MMAs (nine where an accumulator's first product has to be issued on its own), of a pair 128 K of one
// digit of each, in eight. With one box each the issuing thread's wait, descriptors and commit took 560 cycles a stage
// against the 256 of its four MMAs; eight MMAs a stage and descriptors that are additions keep the tensor pipe ahead.
constexpr int kTileM = 128, kTileN = 128, kTileK = 64;
constexpr int kStageBoxes = 2;
constexpr int kStages = 3;
constexpr int kBoxBytes = kTileM * kTileK * 2;               // 16 KB
constexpr int kStageBytes = 2 * kStageBoxes * kBoxBytes;      // A boxes, then B boxes: 64 KB
constexpr int kSlots = 4;                                     // accumulators of 128 tensor-memory columns
constexpr int kTmemCols = kSlots * kTileN;
constexpr int kThreads = 320;                                 // producer, MMA, 8 epilogue warps
constexpr int kMaxGroups = 160;
constexpr int kMaxSlices = 8;
constexpr unsigned kWaitLimit = 1u << 22;  // try_wait rounds before a wait is declared stuck

// One accumulation group over K blocks [kb0, kb0 + nkb). Quads: for p < ni, i = i0 + 2 p, j = d - i, the digit pairs
// (i, j), (i, j + 1), (i + 1, j), (i + 1, j + 1), into three accumulators (diagonals d, d + 1, d + 2). Singles: the
// pairs (i, d - i), i = i0 + step p, into one; step 2 on even diagonals, where quads hold the pairs between.
struct Plan {
    int n_groups;
    int S;
    int s0;  // the int64 accumulator holds the product in units of 2^(-14 - s0) (diagonal d enters times 2^(s0 - 8 (d - 2)))
    unsigned g[kMaxGroups];  // d | i0 << 4 | ni << 8 | kb0 << 12 | nkb << 22 | quads << 31
};
__host__ __device__ inline int g_d(unsigned v) { return v & 15; }
__host__ __device__ inline int g_i0(unsigned v) { return (v >> 4) & 15; }
__host__ __device__ inline int g_ni(unsigned v) { return (v >> 8) & 15; }
__host__ __device__ inline int g_kb0(unsigned v) { return (v >> 12) & 1023; }
__host__ __device__ inline int g_nkb(unsigned v) { return (v >> 22) & 511; }
__host__ __device__ inline bool g_quad(unsigned v) { return v >> 31; }
__host__ __device__ inline int g_step(unsigned v) { return 2 - (int)(v & 1u); }

// ---------------------------------------------------------------- PTX wrappers

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}

// Bounded wait for phase `parity` of bar: false when the CTA is aborting or the wait ran out (which
// starts the abort and records it in *err).
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, volatile int* abort_flag, int* err) {
    for (unsigned it = 0;; ++it) {
        if (mbar_try_wait(bar, parity)) return true;
        if ((it & 63u) == 63u && *abort_flag) return false;
        if (it >= kWaitLimit) {
            *abort_flag = 1;
            atomicOr(err, 1);
            return false;
        }
    }
}

__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* map, int x, int y, int z, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(
            smem_u32(dst)),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(z), "r"(smem_u32(bar))
        : "memory");
}

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// shared-memory matrix descriptor of a K-major tile written by TMA with the 128-byte swizzle: rows of
// 128 bytes, 8-row atoms 1024 bytes apart (stride byte offset), descriptor version 1 (bits 46-48)
__device__ __forceinline__ uint64_t smem_desc_sw128(uint32_t saddr) {
    return (uint64_t)((saddr & 0x3FFFFu) >> 4) | ((uint64_t)1 << 16) | ((uint64_t)(1024 >> 4) << 32) | ((uint64_t)1 << 46) |
           ((uint64_t)2 << 61);
}

// instruction descriptor: D f32, A and B bf16, both K-major, M = 128
__host__ __device__ constexpr uint32_t mma_idesc(int n) { return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(kTileM >> 4) << 24); }

template <int N>
__device__ __forceinline__ void mma_bf16(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t accumulate) {
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}" ::"r"(d_tmem),
        "l"(adesc), "l"(bdesc), "r"(mma_idesc(N)), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void mma_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}

__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float* v) {
    uint32_t r[32];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,"
        "%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]),
          "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]),
          "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int j = 0; j < 32; ++j) v[j] = __uint_as_float(r[j]);
}

// ---------------------------------------------------------------- digit split

// A row of A or column of B holding a non-finite entry gets this exponent: its digits come out zero and
// the epilogue writes NaN for every element of C it touches (any such product is non-finite in FP64 too).
constexpr int kNonFinite = 1 << 20;
// and a zero row or column this one, far below every other: the product's unit is then below any C0, which is kept as it
// is. (With exponent 0 C0 was rounded to 2^-55, whatever its size: a solve lost the rows of a small diagonal block.)
constexpr int kZeroLine = -(1 << 18);

// The split kernels use no FP64 arithmetic: the FP64 pipe of this GPU runs 1/32 of the FP32 rate, and
// conversions between FP64 and 64-bit integers run there too. Magnitudes are compared as the bit patterns
// of |x| (ordered like the values), and a value is brought to fixed point from its exponent and mantissa.
constexpr unsigned long long kMagInf = 0x7FF0000000000000ull;
// |x| as a comparable bit pattern; kMagInf for inf and NaN
__device__ __forceinline__ unsigned long long mag_bits(double x) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(x) & 0x7FFFFFFFFFFFFFFFull;
    return b >= kMagInf ? kMagInf : b;
}

// the scale exponent of a row or column from its largest magnitude's bits: max = f 2^e with f in [0.5, 1);
// kNonFinite when the row or column holds a non-finite entry, kZeroLine when it is zero
__device__ __forceinline__ int scale_exponent(unsigned long long mb) {
    if (mb >= kMagInf) return kNonFinite;
    if (mb == 0) return kZeroLine;
    const int be = (int)(mb >> 52);
    if (be == 0) {  // a subnormal maximum (the FP64 path: rare)
        int e;
        frexp(__longlong_as_double((long long)mb), &e);
        return e;
    }
    return be - 1022;
}

// Y = x 2^(62 - e) rounded to the nearest integer (ties to even), for |x| < 2^e: |Y| < 2^62
__device__ __forceinline__ long long fixed62(double x, int e) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(x);
    const int be = (int)((b >> 52) & 0x7FF);
    if (be == 0) {
        if ((b << 1) == 0) return 0;
        return __double2ll_rn(ldexp(x, 62 - e));  // subnormal: the FP64 path
    }
    const unsigned long long mant = (b & 0xFFFFFFFFFFFFFull) | (1ull << 52);
    const int sh = be - 1075 + 62 - e;  // |Y| = mant 2^sh; |x| < 2^e keeps sh <= 9
    unsigned long long m = 0;
    if (sh >= 0) {
        m = mant << sh;
    } else if (sh > -64) {
        const int r = -sh;
        const unsigned long long rem = mant & ((1ull << r) - 1ull), half = 1ull << (r - 1);
        m = mant >> r;
        if (rem > half || (rem == half && (m & 1ull))) ++m;
    }
    return (b >> 63) ? -(long long)m : (long long)m;
}

// c as an integer count of 2^e2 units (nearest, ties to even), for adding C0 into the accumulator; false when
// c is subnormal, not finite, or at least 2^61 units (the caller adds in FP64 then)
__device__ __forceinline__ bool double_to_units(double c, int e2, long long& t) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(c);
    const int be = (int)((b >> 52) & 0x7FF);
    if (be == 0) {
        t = 0;
        return (b << 1) == 0;
    }
    if (be == 0x7FF) return false;
    const unsigned long long mant = (b & 0xFFFFFFFFFFFFFull) | (1ull << 52);
    const int sh = (be - 1075) - e2;  // c = mant 2^(be - 1075)
    unsigned long long m = 0;
    if (sh >= 0) {
        if (sh > 8) return false;
        m = mant << sh;
    } else if (sh > -64) {
        const int r = -sh;
        const unsigned long long rem = mant & ((1ull << r) - 1ull), half = 1ull << (r - 1);
        m = mant >> r;
        if (rem > half || (rem == half && (m & 1ull))) ++m;
    }
    t = (b >> 63) ? -(long long)m : (long long)m;
    return true;
}

// The digits of x 2^-e (|x 2^-e| < 1), all at once. With Y = |x| 2^(62 - e) rounded to 62 fractional bits, the bytes
// of W = 2 (Y + sum_{s >= 1} 2^(62 - 8 s) + half a unit of the last digit) are the digits of |x| 2^-e: the top byte
// is d_0 in [0, 128] itself and each lower one d_s + 128 with d_s in [-128, 127] (the added 2^(62 - 8 s) are the
// offsets 128; carries have moved up already). Digit s has weight 2^(-7 - 8 s); x's sign goes onto every digit. An
// eighth digit is byte 0. A non-finite x (whose row or column then carries kNonFinite) gives zero digits.
struct DigitWord {
    unsigned hi, lo, sign;  // sign 0x8000 for a negative x
};
// Y of a zero or subnormal x, or one in a row or column with a non-finite entry (out of line: rare)
__device__ __noinline__ unsigned long long digit_y_slow(double x, int e) {
    return mag_bits(x) >= kMagInf || e == kNonFinite ? 0ull : (unsigned long long)fixed62(fabs(x), e);
}
__device__ __forceinline__ unsigned long long digit_offsets(int S) {
    unsigned long long c = 1ull << (54 - 8 * (min(S, 7) - 1));
    for (int s = 1; s < min(S, 7); ++s) c += 1ull << (62 - 8 * s);
    return c;
}
__device__ __forceinline__ DigitWord digit_word(double x, int e, unsigned long long offsets) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(x);
    const int be = (int)((b >> 52) & 0x7FF);
    const unsigned long long mant = ((b & 0xFFFFFFFFFFFFFull) | (1ull << 52)) << 9;  // |x| = mant 2^(be - 1084)
    const int r = min(1022 + e - be, 63);                                           // |x| < 2^e keeps it >= 0
    unsigned long long Y = (mant + ((1ull << (r & 63)) >> 1)) >> (r & 63);
    if (be == 0 || be == 0x7FF || e == kNonFinite) Y = (b << 1) == 0 ? 0ull : digit_y_slow(x, e);
    const unsigned long long W = (Y + offsets) << 1;
    return DigitWord{(unsigned)(W >> 32), (unsigned)W, (unsigned)(b >> 48) & 0x8000u};
}
// digit s of two values as a pair of bf16 (the first in the low half), signs not yet applied: 128 + (byte & 127)
// and 128, 256 or 0 are exact in bf16, and so is their difference
template <int s>
__device__ __forceinline__ unsigned digit_pair(const DigitWord& a, const DigitWord& b) {
    constexpr unsigned byte = s < 4 ? 3 - s : 7 - s;
    const unsigned u = __byte_perm(s < 4 ? a.hi : a.lo, s < 4 ? b.hi : b.lo, byte | (byte + 4) << 8);
    const unsigned x = (u & 0x007f007fu) | 0x43004300u;
    const unsigned c = s == 0 ? 0x43004300u - (u & 0x00800080u) * 0x86u : (u & 0x00800080u) ^ 0x43804380u;
    unsigned d;
    asm("sub.rn.bf16x2 %0, %1, %2;" : "=r"(d) : "r"(x), "r"(c));
    return d;
}
// the S digits of four consecutive values of a row to the planes at out (8-byte aligned), and with a second place
// the same with the signs flipped there if `flip`
template <int s>
__device__ __forceinline__ void store_digit(const DigitWord* w, unsigned sg01, unsigned sg23, uint16_t* out, uint16_t* out2,
                                            unsigned flip, long long plane) {
    const unsigned d01 = digit_pair<s>(w[0], w[1]) ^ sg01, d23 = digit_pair<s>(w[2], w[3]) ^ sg23;
    *reinterpret_cast<uint2*>(out + s * plane) = make_uint2(d01, d23);
    if (out2) *reinterpret_cast<uint2*>(out2 + s * plane) = make_uint2(d01 ^ flip, d23 ^ flip);
}
__device__ __forceinline__ void store_digits4(const double* x, int e, int S, unsigned long long offsets, uint16_t* out, uint16_t* out2,
                                              unsigned flip, long long plane) {
    DigitWord w[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) w[j] = digit_word(x[j], e, offsets);
    // a value that is zero (or in a non-finite row) has all digits zero whatever its sign: -0 times a finite digit is
    // a zero, which the sums ignore
    const unsigned sg01 = w[0].sign | w[1].sign << 16, sg23 = w[2].sign | w[3].sign << 16;
    store_digit<0>(w, sg01, sg23, out, out2, flip, plane);
    if (S > 1) store_digit<1>(w, sg01, sg23, out, out2, flip, plane);
    if (S > 2) store_digit<2>(w, sg01, sg23, out, out2, flip, plane);
    if (S > 3) store_digit<3>(w, sg01, sg23, out, out2, flip, plane);
    if (S > 4) store_digit<4>(w, sg01, sg23, out, out2, flip, plane);
    if (S > 5) store_digit<5>(w, sg01, sg23, out, out2, flip, plane);
    if (S > 6) store_digit<6>(w, sg01, sg23, out, out2, flip, plane);
    if (S > 7) store_digit<7>(w, sg01, sg23, out, out2, flip, plane);
}

// A (m x k, column-major, lda) of matrix blockIdx.y -> S planes of A^ (2m rows x Kp, K contiguous) and
// ea[i]; one CTA per 32 rows of A. Complex B (real_b = 0): rows 2i, 2i+1 = [Re A(i,:), -Im A(i,:)] and
// [Im A(i,:), Re A(i,:)], the second part from Kp / 2 on, zeros after k of each; real B (real_b = 1): rows
// [Re A(i,:)] and [Im A(i,:)] over K = k.
// A is read through a shared-memory tile (coalesced along the rows); a thread then splits four consecutive entries
// of a row and stores them as eight bytes a plane. Bound by integer instructions and the planes' writes: 0.29 us a
// matrix of order 121 (304 of them; 867 KB of planes each, 3.0 TB/s), against 0.90 us of the digit-by-digit form with
// two-byte stores before it.
constexpr int kSplitTile = 32;
__global__ void __launch_bounds__(256) tc_split_a_kernel(int m, int k, int Kp, int S, int real_b, const zc* __restrict__ A,
                                                         int lda, long long a_stride, uint16_t* __restrict__ out,
                                                         int* __restrict__ ea) {
    const long long b = blockIdx.y;
    const int i0 = blockIdx.x * 32, t = threadIdx.x, il = t & 31, w = t >> 5;
    const zc* As = A + b * a_stride;
    __shared__ unsigned long long smax[8][32];
    __shared__ int sexp[32];
    __shared__ zc tile[32][kSplitTile + 1];
    unsigned long long mx = 0;
    if (i0 + il < m) {
#pragma unroll 4
        for (int kk = w; kk < k; kk += 8) {
            const zc v = As[(long long)kk * lda + i0 + il];
            mx = max(mx, max(mag_bits(v.re), mag_bits(v.im)));
        }
    }
    smax[w][il] = mx;
    __syncthreads();
    if (w == 0) {
        for (int q = 1; q < 8; ++q) mx = max(mx, smax[q][il]);
        sexp[il] = scale_exponent(mx);
        if (i0 + il < m) ea[b * m + i0 + il] = sexp[il];
    }
    const long long plane = 2LL * m * Kp;
    uint16_t* o = out + b * S * plane;
    const int half = real_b ? Kp : Kp / 2;
    const unsigned long long offsets = digit_offsets(S);
    const int r = t >> 3, i = i0 + r, q4 = 4 * (t & 7);  // the row and the four columns this thread splits
    for (int kc = 0; kc < half; kc += kSplitTile) {
        __syncthreads();
        for (int q = w; q < kSplitTile; q += 8) {
            const int kk = kc + q;
            tile[il][q] = (kk < k && i0 + il < m) ? As[(long long)kk * lda + i0 + il] : zc{0.0, 0.0};
        }
        __syncthreads();
        if (i >= m) continue;
        const int e = sexp[r];
        double re[4], im[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const zc v = tile[r][q4 + j];
            re[j] = v.re;
            im[j] = v.im;
        }
        uint16_t* row0 = o + 2LL * i * Kp + kc + q4;
        uint16_t* row1 = row0 + Kp;
        store_digits4(re, e, S, offsets, row0, real_b ? nullptr : row1 + half, 0u, plane);
        store_digits4(im, e, S, offsets, row1, real_b ? nullptr : row0 + half, 0x80008000u, plane);
    }
}

// B (k x n, column-major, ldb) -> S planes of B^t (n rows x Kp) and eb[j]; G = 8, 16 or 32 lanes per column (so that
// a k of 32, the factorisations' updates, keeps all lanes busy), four consecutive entries a lane. Complex B:
// [Re B(:, j); Im B(:, j)], the imaginary part from Kp / 2 on; real B (Br, double): B(:, j); zeros after k.
// Order 121 (304 matrices): 0.15 us a matrix against 0.42 us with two-byte stores.
template <int G>
__global__ void __launch_bounds__(128) tc_split_b_kernel(int n, int k, int Kp, int S, int batch, const zc* __restrict__ B,
                                                         const double* __restrict__ Br, int ldb, long long b_stride,
                                                         uint16_t* __restrict__ out, int* __restrict__ eb) {
    const long long gw = ((long long)blockIdx.x * blockDim.x + threadIdx.x) / G;
    if (gw >= (long long)batch * n) return;
    const unsigned mask = group_mask<G>();
    const long long b = gw / n;
    const int j = (int)(gw - b * n), lane = threadIdx.x & (G - 1);
    const zc* col = Br ? nullptr : B + b * b_stride + (long long)j * ldb;
    const double* rcol = Br ? Br + b * b_stride + (long long)j * ldb : nullptr;
    unsigned long long mx = 0;
    if (Br) {
#pragma unroll 4
        for (int kk = lane; kk < k; kk += G) mx = max(mx, mag_bits(rcol[kk]));
    } else {
#pragma unroll 4
        for (int kk = lane; kk < k; kk += G) mx = max(mx, max(mag_bits(col[kk].re), mag_bits(col[kk].im)));
    }
    for (int o = G / 2; o > 0; o >>= 1) mx = max(mx, __shfl_xor_sync(mask, mx, o, G));
    const int e = scale_exponent(mx);
    if (lane == 0) eb[b * n + j] = e;
    const long long plane = (long long)n * Kp;
    uint16_t* o = out + b * S * plane + (long long)j * Kp;
    const unsigned long long offsets = digit_offsets(S);
    const int half = Br ? Kp : Kp / 2;
    for (int kk = 4 * lane; kk < half; kk += 4 * G) {
        double re[4], im[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const bool in = kk + u < k;
            if (Br) {
                re[u] = in ? rcol[kk + u] : 0.0;
            } else {
                const zc v = in ? col[kk + u] : zc{0.0, 0.0};
                re[u] = v.re;
                im[u] = v.im;
            }
        }
        store_digits4(re, e, S, offsets, o + kk, nullptr, 0u, plane);
        if (!Br) store_digits4(im, e, S, offsets, o + kk + half, nullptr, 0u, plane);
    }
}
void split_b(cudaStream_t st, int n, int k, int Kp, int S, int batch, const zc* B, const double* Br, int ldb, long long b_stride,
             uint16_t* out, int* eb) {
    const int half = Br ? Kp : Kp / 2, g = half <= 32 ? 8 : half <= 64 ? 16 : 32;
    const unsigned blocks = (unsigned)(((long long)batch * n * g + 127) / 128);
    if (g == 8) tc_split_b_kernel<8><<<blocks, 128, 0, st>>>(n, k, Kp, S, batch, B, Br, ldb, b_stride, out, eb);
    else if (g == 16) tc_split_b_kernel<16><<<blocks, 128, 0, st>>>(n, k, Kp, S, batch, B, Br, ldb, b_stride, out, eb);
    else tc_split_b_kernel<32><<<blocks, 128, 0, st>>>(n, k, Kp, S, batch, B, Br, ldb, b_stride, out, eb);
    ++launch_count();
}

// ---------------------------------------------------------------- the product

// One element of C from its int64 accumulator ac (units of 2^(e - 14 - s0)), e = ea + eb; NaN for a non-finite row or
// column. With s_ab = +-1 and s_c in {0, 1} (unit_scales, every product of the solves) C0's part joins as an integer
// count of the same unit and the sum is rounded once, to nearest even, by integer operations. (The conversion
// instruction runs on the FP64 pipe: with two warps a scheduler 322 cycles an element against 260.) What is not
// a normal double then, or has other scales, is rare and out of line: inlined, its instructions were issued
// (predicated off) for every element.
__device__ __noinline__ double finish_slow(long long ac, int e, int s0, double c0, double s_ab, double s_c) {
    if (e >= kNonFinite / 2) return __longlong_as_double(0x7FF8000000000000LL);
    return fma(s_c, c0, s_ab * ldexp((double)ac, e - 14 - s0));
}
template <bool HasC0>
__device__ __forceinline__ double finish_fast(long long ac, int e, int s0, long long neg, bool unit_scales, double c0, bool& fast) {
    const int e2 = e - 14 - s0;
    long long a = (ac ^ neg) - neg;  // neg: 0 or -1
    fast = unit_scales;
    if (HasC0) {
        long long t;
        fast = double_to_units(c0, e2, t) && fast;
        a += t;
    }
    const unsigned long long u = (unsigned long long)(a < 0 ? -a : a);  // below 2^63
    const int lz = __clzll((long long)u);
    const unsigned long long w = u << ((lz - 1) & 63);  // the leading one at bit 62
    const unsigned long long q = (w + 0x1FF + ((unsigned)(w >> 10) & 1u)) >> 10;  // 53 bits, or 2^53: the sum below carries it
    const int ex = 1085 - lz + e2;  // biased exponent - 1
    fast = fast && (a == 0 ? e < kNonFinite / 2 : (unsigned)ex < 2045u);
    const int hi = (int)(q >> 32) + (ex << 20) + (a < 0 ? (int)0x80000000 : 0);
    return __hiloint2double(a == 0 ? 0 : hi, a == 0 ? 0 : (int)q);
}
// Four elements at once, their rare cases after all of them: with a branch an element nothing of the next one
// started before the last was done, and two warps a scheduler do not hide that (4096 products of order 121
// with their splits 4.27 to 4.14 ms, of 121 x 32 x 121 1.88 to 1.70, of order 81 3.02 to 2.83).
template <bool HasC0>
__device__ __forceinline__ void finish_four(const long long* ac, const int* e, int s0, long long neg, bool unit_scales, const double* c0,
                                            double s_ab, double s_c, double* out) {
    bool fast[4], all = true;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        out[u] = finish_fast<HasC0>(ac[u], e[u], s0, neg, unit_scales, HasC0 ? c0[u] : 0.0, fast[u]);
        all = all && fast[u];
    }
    if (!all) {
#pragma unroll 1
        for (int u = 0; u < 4; ++u) {
            const bool f = u == 0 ? fast[0] : u == 1 ? fast[1] : u == 2 ? fast[2] : fast[3];
            if (f) continue;
            const long long a = u == 0 ? ac[0] : u == 1 ? ac[1] : u == 2 ? ac[2] : ac[3];
            const int ee = u == 0 ? e[0] : u == 1 ? e[1] : u == 2 ? e[2] : e[3];
            const double c = !HasC0 ? 0.0 : u == 0 ? c0[0] : u == 1 ? c0[1] : u == 2 ? c0[2] : c0[3];
            const double r = finish_slow(a, ee, s0, c, s_ab, HasC0 ? s_c : 0.0);
            if (u == 0) out[0] = r;
            else if (u == 1) out[1] = r;
            else if (u == 2) out[2] = r;
            else out[3] = r;
        }
    }
}

// The accumulator slots of the next group (quads and singles count the groups of each kind so far). Quads need their
// three diagonals in neighbouring columns, the middle one between; they take slots 0 1 2 and 3 2 1 in turn (the
// second with B's boxes exchanged), so that their first products need one slot of the group before, the one that is
// drained first.
struct GroupSlots {
    int low, mid, high;
};
__device__ __forceinline__ GroupSlots group_slots(bool quad, int& quads, int& singles) {
    if (quad) return quads++ & 1 ? GroupSlots{3, 2, 1} : GroupSlots{0, 1, 2};
    const int s = singles++ & 1 ? 0 : 3;
    return GroupSlots{s, s, s};
}

struct SharedState {
    uint64_t full[kStages], empty[kStages], tfull[kSlots], tempty[kSlots], drain;
    uint32_t tmem_base;
    int abort_flag;
    int eb[kTileN];  // the columns' scale exponents
};

// acc += x 2^sh (rounded for sh < 0) for 32 group sums x = v (integers below 2^24; x 2^sh stays below 2^62)
__device__ __forceinline__ void add_group(long long* acc, const float* v, int sh) {
    if (sh >= 32) {
        const int k = sh - 32;
#pragma unroll
        for (int j = 0; j < 32; ++j) acc[j] += (long long)((unsigned long long)(unsigned)(__float2int_rn(v[j]) << k) << 32);
    } else if (sh >= 0) {
        const int dbl = sh == 31, f = 1 << (sh - dbl);
#pragma unroll
        for (int j = 0; j < 32; ++j) {
            const int x = __float2int_rn(v[j]) << dbl;
            asm("mad.wide.s32 %0, %1, %2, %0;" : "+l"(acc[j]) : "r"(x), "r"(f));
        }
    } else {
        const int half = 1 << (-sh - 1);
#pragma unroll
        for (int j = 0; j < 32; ++j) acc[j] += (long long)((__float2int_rn(v[j]) + half) >> -sh);
    }
}

__global__ void __launch_bounds__(kThreads, 1)
    tc_gemm_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b, const __grid_constant__ Plan plan,
                   int m, int n, int batch0, int a_bcast, int b_bcast, const int* __restrict__ ea, const int* __restrict__ eb,
                   const zc* C0, long long c0_stride, zc* C, int ldc, long long c_stride, double s_ab, double s_c,
                   const int* __restrict__ skip, int skip_value, int* __restrict__ err) {
    const int lb = blockIdx.z;  // matrix within this chunk
    if (skip && skip[batch0 + lb] == skip_value) return;
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    SharedState* ss = reinterpret_cast<SharedState*>(smem + kStages * kStageBytes);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int m0 = blockIdx.y * kTileM, n0 = blockIdx.x * kTileN;
    const int S = plan.S;

    if (threadIdx.x == 0) {
        for (int s = 0; s < kStages; ++s) {
            mbar_init(&ss->full[s], 1);
            mbar_init(&ss->empty[s], 1);
        }
        for (int s = 0; s < kSlots; ++s) {
            mbar_init(&ss->tfull[s], 1);
            mbar_init(&ss->tempty[s], 8);
        }
        mbar_init(&ss->drain, 1);
        ss->abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&ss->tmem_base)),
                     "r"(kTmemCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
        tc_fence_before();
    }
    if (warp >= 2 && warp < 6) {
        const int j = threadIdx.x - 64;
        ss->eb[j] = n0 + j < n ? eb[(long long)(b_bcast ? 0 : batch0 + lb) * n + n0 + j] : 0;
    }
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = ss->tmem_base;
    volatile int* abort_flag = &ss->abort_flag;
    const int za = a_bcast ? 0 : lb, zb = b_bcast ? 0 : lb;

    if (warp == 0) {
        // ---- TMA producer
        if (lane == 0) {
            int st = 0, ph = 1, issued = 0, quads = 0;
            bool ok = true;
            for (int gi = 0; gi < plan.n_groups && ok; ++gi) {
                const unsigned g = plan.g[gi];
                const int d = g_d(g), i0 = g_i0(g), ni = g_ni(g), kb0 = g_kb0(g), kb1 = kb0 + g_nkb(g);
                const bool quad = g_quad(g);
                const int step = quad ? 2 : g_step(g), flip = quad ? quads++ & 1 : 0;
                for (int p = 0; p < ni && ok; ++p) {
                    const int i = i0 + step * p, pa = za * S + i - 1, pb = zb * S + d - i - 1;
                    for (int kb = kb0; kb < kb1; kb += quad ? 1 : kStageBoxes) {
                        if (!mbar_wait(&ss->empty[st], ph, abort_flag, err)) {
                            ok = false;
                            break;
                        }
                        unsigned char* sa = smem + st * kStageBytes;
                        uint64_t* full = &ss->full[st];
                        // the second box of each operand: the next digit, or the next K block
                        const int kn = quad ? kb : kb + 1, dn = quad ? 1 : 0;
                        const bool two = quad || kb + 1 < kb1;
                        mbar_expect_tx(full, two ? kStageBytes : kStageBytes / 2);
                        tma_load_3d(sa, &map_a, kb * kTileK, m0, pa, full);
                        tma_load_3d(sa + kStageBoxes * kBoxBytes, &map_b, kb * kTileK, n0, pb + flip, full);
                        if (two) {
                            tma_load_3d(sa + kBoxBytes, &map_a, kn * kTileK, m0, pa + dn, full);
                            tma_load_3d(sa + (kStageBoxes + 1) * kBoxBytes, &map_b, kn * kTileK, n0, pb + dn - flip, full);
                        }
                        ++issued;
                        if (++st == kStages) {
                            st = 0;
                            ph ^= 1;
                        }
                    }
                }
            }
            if (!ok) {
                // drain: wait (bounded) for the copies this thread started into each stage
                for (int s = 0; s < kStages; ++s) {
                    const int uses = (issued + kStages - 1 - s) / kStages;
                    if (uses == 0) continue;
                    for (unsigned r = 0; r < kWaitLimit && !mbar_try_wait(&ss->full[s], (uses - 1) & 1); ++r) {
                    }
                }
            }
        }
    } else if (warp == 1) {
        // ---- MMA issuer
        if (lane == 0) {
            const uint64_t base = smem_desc_sw128(smem_u32(smem));
            int st = 0, ph = 0, quads = 0, singles = 0;
            uint32_t used = 0;  // a bit per slot: the parity of its uses so far
            bool ok = true;
            bool any = false;
            const auto slot_free = [&](int slot) {
                if (!mbar_wait(&ss->tempty[slot], (used >> slot & 1) ^ 1, abort_flag, err)) return false;
                used ^= 1u << slot;
                return true;
            };
            const auto slot_cols = [&](int slot) { return tmem + slot * kTileN; };
            // the four MMAs of one box of A and one of B; descriptors count 16-byte units: 32 bytes of K further is + 2
            const auto box_mma = [&](uint32_t d_tmem, uint64_t da, uint64_t db, uint32_t acc) {
#pragma unroll
                for (int kk = 0; kk < kTileK / 16; ++kk) mma_bf16<kTileN>(d_tmem, da + 2 * kk, db + 2 * kk, kk ? 1u : acc);
            };
            constexpr uint64_t box = kBoxBytes >> 4;
            for (int gi = 0; gi < plan.n_groups && ok; ++gi) {
                const unsigned g = plan.g[gi];
                const int ni = g_ni(g), nkb = g_nkb(g);
                const bool quad = g_quad(g);
                const GroupSlots gs = group_slots(quad, quads, singles);
                uint32_t acc = 0;
                for (int p = 0; p < ni && ok; ++p) {
                    for (int kb = 0; kb < nkb; kb += quad ? 1 : kStageBoxes) {
                        if (!mbar_wait(&ss->full[st], ph, abort_flag, err)) {
                            ok = false;
                            break;
                        }
                        // a slot is waited for when its first product is about to be issued
                        if (!acc && !(slot_free(gs.low) && (!quad || slot_free(gs.mid)))) {
                            ok = false;
                            break;
                        }
                        tc_fence_after();
                        const uint64_t a0 = base + (uint64_t)st * (kStageBytes >> 4), b0 = a0 + kStageBoxes * box;
                        any = true;
                        if (quad) {
                            // A_i by both boxes of B: diagonals d and d + 1, side by side
                            const uint32_t d0 = slot_cols(min(gs.low, gs.mid)), d1 = slot_cols(min(gs.mid, gs.high));
#pragma unroll
                            for (int kk = 0; kk < kTileK / 16; ++kk) mma_bf16<2 * kTileN>(d0, a0 + 2 * kk, b0 + 2 * kk, kk ? 1u : acc);
                            if (!acc) {
                                if (!slot_free(gs.high)) {
                                    ok = false;
                                    break;
                                }
                                tc_fence_after();
                            }
                            // A_(i+1): diagonals d + 1 and d + 2, the first of d + 2 on its own
                            const uint64_t a1 = a0 + box;
                            if (acc) {
                                mma_bf16<2 * kTileN>(d1, a1, b0, 1);
                            } else {
                                mma_bf16<kTileN>(d1, a1, b0, gs.mid < gs.high);
                                mma_bf16<kTileN>(d1 + kTileN, a1, b0 + box, gs.mid > gs.high);
                            }
#pragma unroll
                            for (int kk = 1; kk < kTileK / 16; ++kk) mma_bf16<2 * kTileN>(d1, a1 + 2 * kk, b0 + 2 * kk, 1);
                        } else {
                            box_mma(slot_cols(gs.low), a0, b0, acc);
                            if (kb + 1 < nkb) box_mma(slot_cols(gs.low), a0 + box, b0 + box, 1);
                        }
                        acc = 1;
                        mma_commit(&ss->empty[st]);  // the stage is free once these products have read it
                        if (++st == kStages) {
                            st = 0;
                            ph ^= 1;
                        }
                    }
                }
                if (ok) {
                    mma_commit(&ss->tfull[gs.low]);
                    if (quad) {
                        mma_commit(&ss->tfull[gs.mid]);
                        mma_commit(&ss->tfull[gs.high]);
                    }
                }
            }
            if (!ok && any) {
                // drain: every product issued so far completes before the accumulators are freed
                mma_commit(&ss->drain);
                for (unsigned r = 0; r < kWaitLimit && !mbar_try_wait(&ss->drain, 0); ++r) {
                }
            }
        }
    } else {
        // ---- epilogue: warps 2..9; lane quarter q of tensor memory, column half h
        const int q = warp & 3, h = (warp - 2) >> 2;
        // Every group sum is an integer below 2^24 (exact in the FP32 accumulator). They are added into one
        // int64 per element in units of 2^(-14 - s0): diagonal d enters times 2^(s0 - 8 (d - 2)), exactly
        // while that shift is >= 0, else rounded right (half a unit per group at most); s0 = 47 - log2(Kp)
        // keeps the whole sum below 2^62, so the unit is 2^-53 of the row-and-column scale for K = 256.
        // Integer sums are exact in any order; the element is then (double) acc 2^(ea + eb - 14 - s0), one
        // rounding.
        long long acc[64];
#pragma unroll
        for (int c = 0; c < 64; ++c) acc[c] = 0;
        bool ok = true;
        int quads = 0, singles = 0;
        uint32_t used = 0;
        GroupSlots gs{};
        for (int gi = 0, part = -1; gi < plan.n_groups;) {
            const unsigned g = plan.g[gi];
            if (part < 0) {
                gs = group_slots(g_quad(g), quads, singles);
                part = g_quad(g) ? 2 : 0;
            }
            // the highest diagonal first: its slot is the first that the next quads need
            const int buf = part == 2 ? gs.high : part == 1 ? gs.mid : gs.low;
            ok = mbar_wait(&ss->tfull[buf], used >> buf & 1, abort_flag, err);
            used ^= 1u << buf;
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            tc_fence_after();
            const int sh = plan.s0 - 8 * (g_d(g) + part - 2);
            const uint32_t base = tmem + ((uint32_t)(q * 32) << 16) + buf * kTileN + h * 64;
            float v[32];
            tmem_ld32(base, v);
            add_group(acc, v, sh);
            tmem_ld32(base + 32, v);
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&ss->tempty[buf]);
            add_group(acc + 32, v, sh);
            if (--part < 0) ++gi;
        }
        if (ok && !*abort_flag) {
            // Each lane writes its own row's part of C: row r of C^ is the real (r even) or imaginary part of
            // row r / 2 of C, so a warp's 32 lanes store 32 consecutive doubles of a column. With s_ab = +-1
            // and s_c in {0, 1} (every product of the solves) the element is formed without FP64 arithmetic:
            // C0's part joins the accumulator as an integer count of the same unit, and the sum is rounded
            // once to a double by integer operations; anything else takes the FP64 path.
            const int r = m0 + q * 32 + lane;  // row of A^
            const int i = r >> 1, part = r & 1;
            const int er = (i < m) ? ea[(long long)(a_bcast ? 0 : batch0 + lb) * m + i] : 0;
            double* Cd = reinterpret_cast<double*>(C + (long long)(batch0 + lb) * c_stride);
            const double* C0d = C0 && s_c != 0.0 ? reinterpret_cast<const double*>(C0 + (long long)(batch0 + lb) * c0_stride)
                                                 : nullptr;
            const bool unit_scales = (s_ab == 1.0 || s_ab == -1.0) && (C0d == nullptr || s_c == 1.0);
            // The accumulators go to shared memory first (the stage ring is idle once the last group has
            // landed; column-major by thread, so a warp's accesses are conflict-free), which keeps the
            // conversion loop below out of the registers that hold them.
            long long* sacc = reinterpret_cast<long long*>(smem);
            const int et = threadIdx.x - 64, cols = min(64, n - n0 - h * 64);
#pragma unroll
            for (int c = 0; c < 64; ++c) sacc[c * 256 + et] = acc[c];
            if (i < m) {
                const int* se = ss->eb + h * 64;
                const long long step = 2LL * ldc, neg = s_ab < 0.0 ? -1 : 0;
                long long off2 = 2 * ((long long)(n0 + h * 64) * ldc + i) + part;
                const auto finish = [&](auto has_c0) {
                    constexpr bool kC0 = decltype(has_c0)::value;
                    for (int c = 0; c < cols; c += 4, off2 += 4 * step) {
                        long long ac[4];
                        int e[4];
                        double c0v[4] = {}, r4[4];
#pragma unroll
                        for (int u = 0; u < 4; ++u) {
                            ac[u] = sacc[(c + u) * 256 + et];  // columns past n: zeros
                            e[u] = er + se[c + u];
                            if (kC0 && c + u < cols) c0v[u] = C0d[off2 + u * step];
                        }
                        finish_four<kC0>(ac, e, plan.s0, neg, unit_scales, c0v, s_ab, s_c, r4);
#pragma unroll
                        for (int u = 0; u < 4; ++u)
                            if (c + u < cols) Cd[off2 + u * step] = r4[u];
                    }
                };
                if (C0d) finish(std::true_type{});
                else finish(std::false_type{});
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols) : "memory");
    }
}

// ---------------------------------------------------------------- host side

using EncodeTiled = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                 const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                 CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiled encode_fn() {
    static EncodeTiled fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* f = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &f, 12000, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiled>(f);
    });
    if (!fn) throw EngineError{RCWA_ECUDA, "tensor-core GEMM: cuTensorMapEncodeTiled is not available"};
    return fn;
}

// digit planes (planes x rows x Kp bf16, K contiguous) as a 3-D tensor map with 64 x 128 boxes
CUtensorMap plane_map(const uint16_t* base, long long rows, int Kp, long long planes) {
    CUtensorMap map;
    const cuuint64_t dims[3] = {(cuuint64_t)Kp, (cuuint64_t)rows, (cuuint64_t)planes};
    const cuuint64_t strides[2] = {(cuuint64_t)Kp * 2, (cuuint64_t)rows * Kp * 2};
    const cuuint32_t box[3] = {(cuuint32_t)kTileK, (cuuint32_t)kTileM, 1};
    const cuuint32_t estr[3] = {1, 1, 1};
    const CUresult r = encode_fn()(&map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<uint16_t*>(base), dims, strides,
                                   box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                                   CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) throw EngineError{RCWA_ECUDA, "tensor-core GEMM: tensor map encoding failed"};
    return map;
}

// The groups, smallest contributions first: the single pairs that quads leave (the odd i of the even one of diagonals
// S and S + 1, and all of diagonal S + 1 where S is even), then the quads by their first diagonal. Every accumulator's
// sum is exact in FP32: at most 1024 digit products, so K in chunks of at most 1024 (quads, whose middle diagonal takes
// two pairs each: 512) and as many pairs a group as that leaves.
Plan make_plan(int S, int kblocks) {
    Plan p{};
    p.S = S;
    int lg = 0;
    while ((1 << lg) < kblocks * kTileK) ++lg;
    p.s0 = 47 - lg;
    const auto add = [&](bool quad, int d, int lo, int hi) {  // i = lo, lo + step .. hi
        const int step = quad ? 2 : 2 - (d & 1), most = 1024 / kTileK / (quad ? 2 : 1);
        for (int kb0 = 0; kb0 < kblocks; kb0 += most) {
            const int nkb = std::min(most, kblocks - kb0), per = std::max(1, most / nkb);
            for (int i0 = lo; i0 <= hi; i0 += step * per) {
                if (p.n_groups >= kMaxGroups) throw EngineError{RCWA_EUNSUPPORTED, "tensor-core GEMM: K too large"};
                const int ni = std::min(per, (hi - i0) / step + 1);
                p.g[p.n_groups++] = (unsigned)d | (unsigned)i0 << 4 | (unsigned)ni << 8 | (unsigned)kb0 << 12 | (unsigned)nkb << 22 |
                                    (quad ? 1u << 31 : 0u);
            }
        }
    };
    if (S % 2 == 0) add(false, S + 1, 1, S);
    const int even = S % 2 ? S + 1 : S;
    add(false, even, 1, even - 1);
    for (int d = even - 2; d >= 2; d -= 2) add(true, d, 1, d - 1);
    return p;
}

int* error_flag() { return static_cast<int*>(device_word(1, sizeof(int))); }

}  // namespace

int tc_gemm_slices() {
    static const int s = [] {
        const char* e = std::getenv("RCWA_GB300_TC_SLICES");
        const int v = e ? std::atoi(e) : 7;
        return std::min(kMaxSlices, std::max(2, v));
    }();
    return s;
}

bool tc_gemm_enabled() {
    static const bool on = [] {
        const char* e = std::getenv("RCWA_GB300_GEMM");
        return !(e && std::strcmp(e, "fp64") == 0);
    }();
    return on;
}

namespace {
thread_local int g_fp64_guards = 0;
}
Fp64ProductsGuard::Fp64ProductsGuard() { ++g_fp64_guards; }
Fp64ProductsGuard::~Fp64ProductsGuard() { --g_fp64_guards; }
bool Fp64ProductsGuard::active() { return g_fp64_guards > 0; }

int tc_gemm_error() {
    int h = 0;
    RCWA_CUDA(cudaMemcpy(&h, error_flag(), sizeof(int), cudaMemcpyDeviceToHost));
    return h;
}

namespace {

// C = s_ab A B + s_c C0 with B complex (B) or real (Br)
void tc_product(cudaStream_t st, int m, int n, int k, int batch, const zc* A, int lda, long long a_stride, const zc* B,
                const double* Br, int ldb, long long b_stride, const zc* C0, long long c0_stride, zc* C, int ldc,
                long long c_stride, double s_ab, double s_c, const int* skip, int skip_value) {
    if (batch <= 0 || m <= 0 || n <= 0) return;
    const int smem_bytes = kStages * kStageBytes + 1024 + (int)sizeof(SharedState) + 64;
    ensure_smem_optin(reinterpret_cast<const void*>(tc_gemm_kernel), smem_bytes);
    const int real_b = Br != nullptr;
    const int S = tc_gemm_slices();
    const int kin = real_b ? k : 2 * k;
    const int Kp = ((kin + kTileK - 1) / kTileK) * kTileK;
    const Plan plan = make_plan(S, Kp / kTileK);
    const bool a_bcast = a_stride == 0, b_bcast = b_stride == 0;
    const long long a_bytes = (long long)S * 2 * m * Kp * 2, b_bytes = (long long)S * n * Kp * 2;
    // matrices per pass: digit planes of at most ~1 GiB
    const long long per = (a_bcast ? 0 : a_bytes) + (b_bcast ? 0 : b_bytes) + 1;
    const int chunk = (int)std::max(1LL, std::min<long long>(batch, (1LL << 30) / per));
    int* err = error_flag();

    const int na = a_bcast ? 1 : chunk, nb = b_bcast ? 1 : chunk;
    DeviceScratch mem(st);
    uint16_t *pa = mem.get<uint16_t>((size_t)a_bytes / 2 * na), *pb = mem.get<uint16_t>((size_t)b_bytes / 2 * nb);
    int *dea = mem.get<int>((size_t)m * (a_bcast ? 1 : batch)), *deb = mem.get<int>((size_t)n * (b_bcast ? 1 : batch));
    const CUtensorMap map_a = plane_map(pa, 2LL * m, Kp, (long long)na * S);
    const CUtensorMap map_b = plane_map(pb, n, Kp, (long long)nb * S);
    if (a_bcast) {
        tc_split_a_kernel<<<dim3((m + 31) / 32, 1), 256, 0, st>>>(m, k, Kp, S, real_b, A, lda, 0, pa, dea);
        ++launch_count();
    }
    if (b_bcast) {
        split_b(st, n, k, Kp, S, 1, B, Br, ldb, 0, pb, deb);
    }
    for (int b0 = 0; b0 < batch; b0 += chunk) {
        const int cb = std::min(chunk, batch - b0);
        if (!a_bcast) {
            tc_split_a_kernel<<<dim3((m + 31) / 32, cb), 256, 0, st>>>(m, k, Kp, S, real_b, A + (long long)b0 * a_stride, lda,
                                                                        a_stride, pa, dea + (long long)b0 * m);
            ++launch_count();
        }
        if (!b_bcast) {
            split_b(st, n, k, Kp, S, cb, B ? B + (long long)b0 * b_stride : nullptr, Br ? Br + (long long)b0 * b_stride : nullptr, ldb,
                    b_stride, pb, deb + (long long)b0 * n);
        }
        const dim3 grid((n + kTileN - 1) / kTileN, (2 * m + kTileM - 1) / kTileM, cb);
        tc_gemm_kernel<<<grid, kThreads, smem_bytes, st>>>(map_a, map_b, plan, m, n, b0, a_bcast, b_bcast, dea, deb, C0,
                                                           c0_stride, C, ldc, c_stride, s_ab, s_c, skip, skip_value, err);
        ++launch_count();
        RCWA_CUDA(cudaGetLastError());
    }
}

}  // namespace

void launch_zgemm_tc(cudaStream_t st, int m, int n, int k, int batch, const zc* A, int lda, long long a_stride,
                     const zc* B, int ldb, long long b_stride, const zc* C0, long long c0_stride, zc* C, int ldc,
                     long long c_stride, double s_ab, double s_c, const int* skip, int skip_value) {
    tc_product(st, m, n, k, batch, A, lda, a_stride, B, nullptr, ldb, b_stride, C0, c0_stride, C, ldc, c_stride, s_ab, s_c,
               skip, skip_value);
}

void launch_zdgemm_tc(cudaStream_t st, int m, int n, int k, int batch, const zc* A, int lda, long long a_stride,
                      const double* B, int ldb, long long b_stride, zc* C, int ldc, long long c_stride, const int* skip,
                      int skip_value) {
    tc_product(st, m, n, k, batch, A, lda, a_stride, nullptr, B, ldb, b_stride, nullptr, 0, C, ldc, c_stride, 1.0, 0.0,
               skip, skip_value);
}

}  // namespace rcwa_gb300
