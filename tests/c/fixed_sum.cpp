// The fixed-point sums' arithmetic (csrc/fixed_sum.cuh) compiled for the host:
// n addends' limbs, their sums, the value read from them.  -ffp-contract=off
// gives the device's single operations.
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>

#define __device__
#define __forceinline__ inline

template <class To, class From>
static To bits_of(From f) {
    static_assert(sizeof(To) == sizeof(From), "");
    To t;
    memcpy(&t, &f, sizeof(t));
    return t;
}
static uint32_t __float_as_uint(float f) { return bits_of<uint32_t>(f); }
static int __float_as_int(float f) { return bits_of<int>(f); }
static float __uint_as_float(uint32_t u) { return bits_of<float>(u); }
static long long __double_as_longlong(double d) { return bits_of<long long>(d); }
static double __longlong_as_double(long long l) { return bits_of<double>(l); }
static int __double2hiint(double d) { return (int)(bits_of<long long>(d) >> 32); }
static float __fadd_rn(float a, float b) { return a + b; }
static float __fsub_rn(float a, float b) { return a - b; }
static float __fmul_rn(float a, float b) { return a * b; }
static float __int2float_rn(int i) { return (float)i; }
static int __float2int_rn(float f) { return (int)lrintf(f); }
static double __ll2double_rn(long long l) { return (double)l; }
static int __clzll(long long l) { return l ? __builtin_clzll((unsigned long long)l) : 64; }
using std::max;
using std::min;

namespace nbg {
struct FF {
    float hi, lo;
};
static FF fast_two_sum(float a, float b) {
    const float s = a + b;
    return {s, b - (s - a)};
}
}  // namespace nbg

#include "fixed_sum.cuh"

using namespace nbg;

// Both return 1 where the sum has to be taken another way.
extern "C" int sum_ff(int n, const float* hi, const float* lo, float last, float* out) {
    const float scale = window_scale(last);
    long long total[kSumWords] = {0};
    for (int i = 0; i < n; i++) {
        int l[kSumWords];
        limbs_of(FF{hi[i], lo[i]}, scale, l);
        for (int j = 0; j < kSumWords; j++) total[j] += l[j];
    }
    long long x;
    int e;
    const bool bad = read_limbs(total, window_exponent(scale), kLeastFF, x, e);
    if (bad) return 1;
    const FF f = exact_ff(x, e);
    out[0] = f.hi;
    out[1] = f.lo;
    return 0;
}

extern "C" int sum_f64(int n, const double* v, double last, double* out) {
    const int E = window_f64(last);
    long long total[kSumWords] = {0};
    for (int i = 0; i < n; i++) {
        int l[kSumWords];
        limbs_of(v[i], E, l);
        for (int j = 0; j < kSumWords; j++) total[j] += l[j];
    }
    long long x;
    int e;
    if (read_limbs(total, E, kLeastF64, x, e)) return 1;
    *out = exact_f64(x, e);
    return 0;
}

// Whether the grid chosen for `blocks` blocks counts itself: each adds one to the
// top byte of a word that may hold anything before.
extern "C" int grid_counts(unsigned blocks, unsigned long long before) {
    const unsigned G = exact_grid(blocks);
    unsigned long long d = before;
    for (unsigned b = 0; b < G; b++) d += 1ull << 56;
    return G >= 1 && G <= blocks && (d - before) >> 56 == G;
}
