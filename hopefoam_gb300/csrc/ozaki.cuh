// ozaki.cuh -- FP64 matrix products on the 16-bit tensor cores by error-free
// slicing (Ootomo, Ozaki and Yokota, "DGEMM on integer matrix multiplication
// unit", and Mukunoki et al., "DGEMM using tensor cores": the Ozaki scheme).
//
// Every row of an operand is held as fixed-point numbers under one power of
// two, W = v 2^(63 - E) (truncated) with |v| < 2^E for the whole row, and W is cut
// into seven signed base-256 digits (56 bits):
//   v = sum_i a_i 2^(E - 7 - 8 i),   a_i in [-128, 127].
// Digits are exact in FP16, digit products are below 2^14, and a sum of up
// to 2^24 / 2^14 of them is exact in the tensor core's FP32 accumulator.  With
// D_s the accumulator of all digit pairs i + j = s,
//   sum_k a[k] b[k] = sum_s D_s 2^(EA + EB - 14 - 8 s),
// which is summed in 64-bit integers and rounded once to FP64.  Against an
// FMA chain this trades the rounding of every partial sum for the truncation
// of the digits past the seventh (both near 2^-55 of the largest product).
//
// GB300 retires two FP64 operations per clock per SM, so the conversions are
// integer code as well (none of them touches the FP64 pipe).  The integer
// parts compile for the host: the operator images are built and the
// conversions checked there.
#pragma once

#include <cstdint>
#include <cstring>

#ifdef __CUDACC__
#include <cuda_fp16.h>
#define OZ_HD __host__ __device__ __forceinline__
#else
#define OZ_HD inline
#endif

namespace oz {

constexpr int kSlices = 7;

OZ_HD uint64_t d_bits(double v) {
#ifdef __CUDA_ARCH__
    return (uint64_t)__double_as_longlong(v);
#else
    uint64_t u;
    memcpy(&u, &v, 8);
    return u;
#endif
}

OZ_HD double bits_d(uint64_t u) {
#ifdef __CUDA_ARCH__
    return __longlong_as_double((long long)u);
#else
    double v;
    memcpy(&v, &u, 8);
    return v;
#endif
}

// high word of |v|: its order is the order of the magnitudes to 2^-20
OZ_HD uint32_t mag_hi(double v) { return (uint32_t)(d_bits(v) >> 32) & 0x7FFFFFFFu; }

// biased exponent bound eb of a row whose largest magnitude has high word
// `maxhi`: |v| + 2^(E - 8) (1 + 2^-7) < 2^E, E = eb - 1022.  The margin keeps the leading
// digit of W inside [-128, 127] after rounding.  Infinite and NaN rows give
// eb >= 2047; a zero row gives 0.
OZ_HD int row_bound(uint32_t maxhi) { return (int)((maxhi + 0x2030u) >> 20); }

// rows outside these bounds are left to plain FP64 arithmetic (their scaled
// exponents could leave the FP64 range); a row of zeros is fine
OZ_HD bool row_ok(uint32_t maxhi) {
    const int eb = row_bound(maxhi);
    return maxhi == 0u || (eb > 300 && eb < 1700);
}

// W + 0x8080808080808080: byte 7 - i is digit i plus 128 (the constant both
// biases the digits and rounds at the seventh).  v must be inside the row's
// bound; subnormal values count as 0.
OZ_HD uint64_t biased(double v, int eb) {
    const uint64_t b = d_bits(v);
    const uint32_t hi = (uint32_t)(b >> 32), lo = (uint32_t)b;
    const int e = (int)((hi >> 20) & 0x7FFu);
    const uint32_t mh = (hi & 0xFFFFFu) | (e ? 0x100000u : 0u);
    uint32_t wh, wl;
    int d = eb - e;
#ifdef __CUDA_ARCH__
    d = d > 63 ? 63 : d;
    wh = __funnelshift_l(lo, mh, 10);
    wl = lo << 10;
    if (d & 32) {
        wl = wh;
        wh = 0u;
    }
    wl = __funnelshift_r(wl, wh, d);
    wh >>= (d & 31);
    if (e == 0) wl = wh = 0u;
#else
    uint64_t w = (((uint64_t)mh << 32) | lo) << 10;
    w = (e == 0 || d > 63 || d < 0) ? 0 : w >> d;
    wh = (uint32_t)(w >> 32);
    wl = (uint32_t)w;
#endif
    const uint64_t w64 = ((uint64_t)wh << 32) | wl;
    const uint64_t s = (uint64_t)(int64_t)((int32_t)hi >> 31);
    return (w64 ^ s) - s + 0x8080808080808080ull;
}

OZ_HD int digit(uint64_t y, int i) { return (int)((y >> (56 - 8 * i)) & 255u) - 128; }

// Z 2^ex, rounded to nearest (ties away); ex and Z keep the result normal
OZ_HD double from_fixed(int64_t Z, int ex) {
    const uint64_t s = (uint64_t)(Z >> 63);
    const uint64_t m = ((uint64_t)Z ^ s) - s;
#ifdef __CUDA_ARCH__
    const int lz = __clzll((long long)m);
#else
    const int lz = m ? __builtin_clzll(m) : 64;
#endif
    const uint64_t n = m << (lz & 63);
    const uint64_t r = (n >> 11) + ((n >> 10) & 1u);
    const uint64_t q = r + ((uint64_t)(uint32_t)(1085 - lz + ex) << 52);
    return m == 0 ? 0.0 : bits_d(q | (s & 0x8000000000000000ull));
}

// Eight accumulators (pairs i + j <= 7) of a nodal product, each below 2^22 in
// magnitude: the base-256 digits of 2^32 hi + lo.  Z = 2^20 hi + lo / 2^12 is the
// sum times 2^(58 - EA - EB): it fits 63 bits when sum |b| < 32 2^EB over the row
// of b.
OZ_HD double combine_nodal(int d0, int d1, int d2, int d3, int d4, int d5, int d6, int d7, int ebab) {
    const int64_t hi = (int64_t)(d0 * 256 + d1) * 65536 + (d2 * 256 + d3);
    const int64_t lo = (int64_t)(d4 * 256 + d5) * 65536 + (d6 * 256 + d7);
    return from_fixed((hi << 20) + (lo >> 12), ebab - 2044 - 58);
}

// the same without the last group
OZ_HD double combine7(int d0, int d1, int d2, int d3, int d4, int d5, int d6, int ebab) {
    return combine_nodal(d0, d1, d2, d3, d4, d5, d6, 0, ebab);
}

// eight accumulators of a flux product, each below 2^24; Z is the sum times
// 2^(56 - EA - EB) and fits when sum |b| < 128 2^EB.  ebab: the biased bounds
// of both rows added.
OZ_HD double combine8(const int* d, int ebab) {
    const int64_t hi = (int64_t)(d[0] * 256 + d[1]) * 65536 + ((int64_t)d[2] * 256 + d[3]);
    const int64_t lo = ((int64_t)d[4] * 256 + d[5]) * 65536 + ((int64_t)d[6] * 256 + d[7]);
    return from_fixed((hi << 18) + (lo >> 14), ebab - 2044 - 56);
}

// FP16 bits of a digit
OZ_HD uint16_t half_bits(int d) {
    if (d == 0) return 0;
    const uint16_t s = d < 0 ? 0x8000u : 0u;
    const unsigned m = (unsigned)(d < 0 ? -d : d);
    int e = 0;
    while ((m >> (e + 1)) != 0) e++;
    return (uint16_t)(s | ((unsigned)(15 + e) << 10) | ((m << (10 - e)) & 0x3FFu));
}

#ifdef __CUDACC__
// digit i of two values as an FP16 pair (a in the low half): 1024 + byte is
// exact in FP16, and so is the difference with 1024 + 128
__device__ __forceinline__ uint32_t digit_pair(uint64_t ya, uint64_t yb, int i) {
    const uint32_t wa = i < 4 ? (uint32_t)(ya >> 32) : (uint32_t)ya;
    const uint32_t wb = i < 4 ? (uint32_t)(yb >> 32) : (uint32_t)yb;
    const unsigned b = (unsigned)((7 - i) & 3);
    uint32_t t = __byte_perm(wa, wb, b | (b << 4) | ((4 + b) << 8) | ((4 + b) << 12));
    t = (t & 0x00FF00FFu) | 0x64006400u;
    __half2 h;
    memcpy(&h, &t, 4);
    h = __hadd2(h, __half2(__ushort_as_half(0xE480), __ushort_as_half(0xE480)));  // - 1152
    memcpy(&t, &h, 4);
    return t;
}

// accumulator to integer: |x| < 2^22 (one FP32 addition) and |x| < 2^24
__device__ __forceinline__ int acc_int22(float x) { return __float_as_int(x + 12582912.f) - 0x4B400000; }
__device__ __forceinline__ int acc_int24(float x) { return __float2int_rn(x); }

// 1 / x and sqrt(x) from an FP32 seed by one cubic step each (Householder's
// iteration of order two; the seed is good to 2^-21, the step to 2^-63)
__device__ __forceinline__ double seed_of(float y) {
    const uint32_t u = __float_as_uint(y);
    const uint32_t e = (u >> 23) & 0xFFu;
    const uint32_t h = (e == 0u || e == 255u) ? 0x7FF80000u : (u & 0x80000000u) | ((e + 896u) << 20) | ((u & 0x7FFFFFu) >> 3);
    return __hiloint2double((int)h, (int)(u << 29));
}
__device__ __forceinline__ float trunc32(double q) {  // 0 or infinite outside the FP32 range
    const uint32_t H = (uint32_t)__double2hiint(q), Lw = (uint32_t)__double2loint(q);
    const uint32_t e = (H >> 20) & 0x7FFu;
    const uint32_t f = (H & 0x80000000u) | ((e - 896u) << 23) | ((H & 0xFFFFFu) << 3) | (Lw >> 29);
    return e < 897u ? 0.f : e > 1150u ? __uint_as_float(0x7F800000u) : __uint_as_float(f);
}
// outside the FP32 range these give NaN (the caller's plain FP64 route takes such elements)
__device__ __forceinline__ double rcp64(double x) {
    float y;
    asm("rcp.approx.f32 %0, %1;" : "=f"(y) : "f"(trunc32(x)));
    const double r = seed_of(y);
    const double e = fma(-x, r, 1.0);
    return fma(r, fma(e, e, e), r);
}
__device__ __forceinline__ double rsqrt64(double x) {
    float y;
    asm("rsqrt.approx.f32 %0, %1;" : "=f"(y) : "f"(trunc32(x)));
    const double r = seed_of(y);
    const double t = x * r;
    const double e = fma(-t, r, 1.0);
    return fma(r * e, fma(0.375, e, 0.5), r);
}
__device__ __forceinline__ double sqrt64(double x) {
    float y;
    asm("rsqrt.approx.f32 %0, %1;" : "=f"(y) : "f"(trunc32(x)));
    const double r = seed_of(y);
    const double t = x * r;
    const double e = fma(-t, r, 1.0);
    return fma(t * e, fma(0.375, e, 0.5), t);
}
#endif

}  // namespace oz
