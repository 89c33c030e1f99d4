// Host stand-ins for the CUDA names the fixed-point eigensolver uses, with warps: every emulated thread of a
// CTA is a fiber (ucontext), warp primitives meet the 32 fibers of a warp and __syncthreads all of them, so
// code in which the warps of a CTA do different things runs as on the device. One CTA at a time; shared
// arrays are statics. Test infrastructure only; it emulates semantics, not performance.
#pragma once
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstdlib>
#include <cstring>

#define __host__
#define __device__
#define __forceinline__ inline
#define __global__
#define __launch_bounds__(x)
#define __align__(x) alignas(x)
#define __restrict__
#define __shared__ static
#define RCWA_DYN_SMEM(T, name) T* const name = reinterpret_cast<T*>(emu_smem)

using std::max;
using std::min;
struct dim3e {
    unsigned x, y = 0, z = 0;
};
extern dim3e threadIdx, blockIdx, blockDim;
extern unsigned char* emu_smem;
struct int2 {
    int x, y;
};
struct double2 {
    double x, y;
};
struct int4 {
    int x, y, z, w;
};
inline int4 make_int4(int a, int b, int c, int d) { return {a, b, c, d}; }
inline double2 make_double2(double a, double b) { return {a, b}; }
inline int2 make_int2(int a, int b) { return {a, b}; }
template <class To, class From>
inline To emu_bits(From f) {
    static_assert(sizeof(To) == sizeof(From));
    To t;
    std::memcpy(&t, &f, sizeof t);
    return t;
}
inline double __longlong_as_double(long long v) { return emu_bits<double>(v); }
inline long long __double_as_longlong(double v) { return emu_bits<long long>(v); }
inline int __float_as_int(float v) { return emu_bits<int>(v); }
inline float __int_as_float(int v) { return emu_bits<float>(v); }
inline int __clz(int v) { return v ? __builtin_clz((unsigned)v) : 32; }
inline int __clzll(long long v) { return v ? __builtin_clzll((unsigned long long)v) : 64; }
inline int __ffs(unsigned x) { return __builtin_ffs((int)x); }
inline unsigned long long __umul64hi(unsigned long long a, unsigned long long b) {
    return (unsigned long long)(((unsigned __int128)a * b) >> 64);
}
inline double rsqrt(double x) { return 1.0 / std::sqrt(x); }
inline float rsqrtf(float x) { return 1.0f / std::sqrt(x); }

void emu_block_sync();
void emu_warp_sync();
extern uint64_t emu_slot[1024];
inline void __syncthreads() { emu_block_sync(); }
inline void __syncwarp(unsigned = 0xffffffffu) { emu_warp_sync(); }
template <class T>
inline T emu_exchange(T v, unsigned from) {  // from: a lane of this warp
    static_assert(sizeof(T) <= 8);
    std::memcpy(&emu_slot[threadIdx.x], &v, sizeof v);
    emu_warp_sync();
    T r;
    std::memcpy(&r, &emu_slot[(threadIdx.x & ~31u) + (from & 31u)], sizeof r);
    emu_warp_sync();
    return r;
}
template <class T>
inline T __shfl_sync(unsigned, T v, int src, int = 32) { return emu_exchange(v, (unsigned)src); }
template <class T>
inline T __shfl_xor_sync(unsigned, T v, int o, int = 32) { return emu_exchange(v, (threadIdx.x & 31u) ^ (unsigned)o); }
template <class T>
inline T __shfl_down_sync(unsigned, T v, int d, int = 32) {
    const unsigned l = threadIdx.x & 31u;
    return emu_exchange(v, l + d < 32 ? l + d : l);
}
inline unsigned __ballot_sync(unsigned, int pred) {
    emu_slot[threadIdx.x] = pred != 0;
    emu_warp_sync();
    unsigned b = 0;
    for (unsigned k = 0; k < 32; ++k)
        if (emu_slot[(threadIdx.x & ~31u) + k]) b |= 1u << k;
    emu_warp_sync();
    return b;
}
inline unsigned long long atomicMax(unsigned long long* p, unsigned long long v) {
    const unsigned long long o = *p;
    *p = std::max(o, v);
    return o;
}
inline unsigned long long atomicAdd(unsigned long long* p, unsigned long long v) {
    const unsigned long long o = *p;
    *p += v;
    return o;
}
