// The arithmetic of the fixed-point sums (allreduce.cuh): a value's limbs, a
// sum's value from the sums of its addends' limbs.  Integer and single
// floating-point operations of one thread, so that a host program can compile
// it too (tests/c/fixed_sum.cpp).
#pragma once

#ifdef __CUDACC__
#include "common.cuh"
#endif

namespace nbg {

constexpr int kLimbs = 5, kLimbBits = 20;
constexpr int kSumWords = kLimbs + 1;  // per value: the limbs, values outside the window
// Blocks of a launch that sums in fixed point: they are counted in the top byte of
// a word, and a count past 255 would never be complete.
constexpr unsigned kExactMaxBlocks = 255;
constexpr unsigned exact_grid(unsigned blocks) {
    return blocks < kExactMaxBlocks ? blocks : kExactMaxBlocks;
}

// 2^-E for the window |v| < 2^E of a sum whose last value was `last` (0:
// none): E = 20 + its exponent.
__device__ __forceinline__ float window_scale(float last) {
    const int ex = (int)((__float_as_uint(last) >> 23) & 255u) - 127;
    if (ex < -80 || ex > 80) return 0.f;  // zero, tiny, huge, not finite
    return __uint_as_float((uint32_t)(127 - ex - kLimbBits) << 23);
}

__device__ __forceinline__ int window_exponent(float scale) {
    return 127 - (int)(__float_as_uint(scale) >> 23);
}

// Limbs of a float-float value: adding 1.5 2^23 units rounds to the unit.
__device__ __forceinline__ void limbs_of(FF v, float scale, int (&l)[kSumWords]) {
    float h = __fmul_rn(v.hi, scale), c = __fmul_rn(v.lo, scale);
    const bool out = !(fabsf(h) < 1.f && fabsf(c) < 1.f) || scale == 0.f;
    if (out) h = c = 0.f;
    l[kLimbs] = out;
#pragma unroll
    for (int j = 0; j < kLimbs; j++) {
        const float m = __uint_as_float((uint32_t)(127 + 23 - kLimbBits * (j + 1)) << 23 | 0x400000u);
        const float th = __fadd_rn(h, m), tc = __fadd_rn(c, m);
        l[j] = (__float_as_int(th) - __float_as_int(m)) + (__float_as_int(tc) - __float_as_int(m));
        h = __fsub_rn(h, __fsub_rn(th, m));
        c = __fsub_rn(c, __fsub_rn(tc, m));
    }
}

// E of the window |v| < 2^E for an FP64 sum whose last value was `last`;
// kNoWindow: none.
constexpr int kNoWindow = -100000;
__device__ __forceinline__ int window_f64(double last) {
    const int ex = (int)((__double2hiint(last) >> 20) & 2047) - 1023;
    return ex < -300 || ex > 300 ? kNoWindow : ex + kLimbBits;
}

// Limbs of an FP64 value: its significand shifted to units of 2^(E - 100),
// rounded there.
__device__ __forceinline__ void limbs_of(double v, int E, int (&l)[kSumWords]) {
    const long long bits = __double_as_longlong(v);
    const int ex = (int)(bits >> 52) & 2047;
    const bool out = E == kNoWindow || ex == 2047 || ex - 1023 >= E;
    unsigned long long m = (unsigned long long)bits & ((1ull << 52) - 1) | 1ull << 52;
    // subnormal values and those that a right shift clears count as zero:
    // 2^-80 of the last sum at most
    int sh = ex - 1075 - E + kLimbs * kLimbBits;
    if (out || ex == 0 || sh < -53) {
        m = 0;
        sh = 0;
    }
    unsigned long long lo, hi = 0;
    if (sh < 0) {
        lo = (m + (1ull << (-sh - 1))) >> -sh;
    } else {
        lo = m << sh;
        hi = sh ? m >> (64 - sh) : 0;
    }
    constexpr int kMask = (1 << kLimbBits) - 1;
    const int s = bits < 0 ? -1 : 1;
    l[4] = s * (int)(lo & kMask);
    l[3] = s * (int)(lo >> 20 & kMask);
    l[2] = s * (int)(lo >> 40 & kMask);
    l[1] = s * (int)((lo >> 60 | hi << 4) & kMask);
    l[0] = s * (int)(hi >> 16);
    l[kLimbs] = out;
}

// The least exponent e of a sum x 2^e that exact_ff (exact_f64) reads: 2^(e + 31)
// is a normal float.  A float-float sum then is at least 2^-97, below which its
// low part would have no bits left.
constexpr int kLeastFF = -126 - 31, kLeastF64 = -1000;

// A sum's value from the sums l of its addends' limbs: an integer x of 61 bits
// and an exponent e, x 2^e.  window: the exponent E of its limbs; least: of kLeastFF
// and kLeastF64 the one that the sum is read as.  True: outside the window, to be
// summed another way.
__device__ __forceinline__ bool read_limbs(const long long (&l)[kSumWords], int window, int least,
                                           long long& x, int& e) {
    // carries: hi 2^60 + lo 2^20 + l4 units of 2^(E - 100)
    const long long l4 = l[4] & ((1 << kLimbBits) - 1);
    long long lo = (l[2] << kLimbBits) + l[3] + (l[4] >> kLimbBits);
    const long long hi = (l[0] << kLimbBits) + l[1] + (lo >> 40);
    lo &= (1ll << 40) - 1;
    // the leading 61 bits: m bits of the last limb (m < 0: bits of lo dropped)
    const int used = 64 - __clzll(hi < 0 ? ~hi : hi);
    const int m = min(21 - used, kLimbBits);
    long long v;
    if (m >= 0) v = (hi << (40 + m)) + (lo << m) + (l4 >> (kLimbBits - m));
    else v = m >= -40 ? (hi << (40 + m)) + (lo >> -m) : hi >> (-m - 40);
    // every addend is rounded to half a unit: n addends to n 2^-57 of a sum that is
    // 2^24 times below the last one, under the bound of a sum by FP64 adds (n 2^-53);
    // a smaller one has too few bits left
    const bool few = m == kLimbBits && (v < 0 ? -v : v) < (1ll << 56);
    const int up = max(__clzll(v < 0 ? ~v : v) - 3, 0);
    x = v << up;
    e = window - 4 * kLimbBits - m - up;
    return l[kLimbs] != 0 || few || e < least;
}

// x 2^e in FP64.
__device__ __forceinline__ double exact_f64(long long x, int e) {
    if (x == 0) return 0.0;
    return __longlong_as_double(__double_as_longlong(__ll2double_rn(x)) + ((long long)e << 52));
}

// x 2^e as a float-float number (|x| < 2^61, e >= kLeastFF): the leading 31 bits and the 31 below them, each exact in an
// integer register.
__device__ __forceinline__ FF exact_ff(long long x, int e) {
    const int a = (int)(x >> 31);
    const float h = __int2float_rn(a);
    const int b = ((a - __float2int_rn(h)) << 24) + ((int)x >> 7 & 0xffffff);
    const float s = __uint_as_float((uint32_t)(e + 31 + 127) << 23);
    return fast_two_sum(__fmul_rn(h, s), __fmul_rn(__fmul_rn(__int2float_rn(b), 0x1p-24f), s));
}

}  // namespace nbg
