// FP64 dot products on the integer pipes, for contractions that FP64 issue would bound.
//
// GB300 issues two FP64 instructions per SM and clock, but 61 32 x 32 + 64 -> 64 bit multiply-adds
// (measured: 0.62 T against 18.1 T a second). A vector of doubles is brought to one exponent and held
// as 84-bit two's-complement integers in three limbs of 28 bits; a product of two of them, to 2^-82 of
// the largest possible one, is six such multiply-adds into three 64-bit sums, in which up to 42
// products fit without a carry. So a dot product costs a fifth of an FP64 one in issue time, and
// nothing is rounded until its end.
//
// Accuracy. With S = 2^(emax - 1022) of each vector, an entry is cut at 2^-84 S (a double has 53 bits, so
// entries within 2^31 of the largest are held exactly) and a product at 2^-82 of the two vectors' S. That
// says nothing about a result whose terms are all far below the product of the largest entries (a large
// entry may meet only small ones), so limbs carry their entry's exponent and the caller forms the largest
// exponent of the terms that a result does have. Where it lies too far below the vectors' (the caller
// states the bound), or a value is infinite, NaN or near the ends of the exponent range, the caller takes
// its FP64 path.
#pragma once

#include <cstdint>

#include <cuda_runtime.h>

namespace gfgpu {

constexpr uint32_t kFxMask = (1u << 28) - 1u;

// biased exponent of a double (0 for zeros and subnormals, 0x7ff for infinities and NaN)
__device__ __forceinline__ int fx_exponent(double d)
{
    return (__double2hiint(d) >> 20) & 0x7ff;
}

// what a zero has in the place of an exponent: below 0 with any two exponents added
constexpr int kFxNone = -(1 << 14);

// d / 2^(emax - 1022) as limbs {x, y, z}: x 2^-28 + y 2^-56 + z 2^-84, emax >= the exponent of d, and in w
// the exponent (1 for a subnormal, kFxNone for a zero); subnormals count as zero (they lie below the cut
// of any vector the caller may pass)
__device__ __forceinline__ int4 fx_from_double(double d, int emax)
{
    const uint32_t hi = static_cast<uint32_t>(__double2hiint(d)), lo = static_cast<uint32_t>(__double2loint(d));
    const int e = static_cast<int>((hi >> 20) & 0x7ffu);
    // 53-bit significand at the top of 96 bits w2:w1:0
    uint32_t w2 = e ? (0x80000000u | (hi << 11) | (lo >> 21)) : 0u, w1 = e ? lo << 11 : 0u, w0 = 0u;
    uint32_t s = static_cast<uint32_t>(emax - e) + 12u; // 84 bits remain of the 96 for e = emax
    if (s >= 64u) {
        w0 = w2;
        w1 = 0u;
        w2 = 0u;
        s -= 64u;
    }
    else if (s >= 32u) {
        w0 = w1;
        w1 = w2;
        w2 = 0u;
        s -= 32u;
    }
    s = min(s, 32u);
    const uint32_t r0 = __funnelshift_rc(w0, w1, s), r1 = __funnelshift_rc(w1, w2, s);
    const uint32_t r2 = s < 32u ? w2 >> s : 0u;
    const int sg = static_cast<int>(hi) >> 31 | 1; // +-1
    return make_int4(static_cast<int>(__funnelshift_l(r1, r2, 8)) * sg,
                     static_cast<int>(__funnelshift_l(r0, r1, 4) & kFxMask) * sg, static_cast<int>(r0 & kFxMask) * sg,
                     e ? e : (((hi << 1) | lo) ? 1 : kFxNone));
}

// sum of products: a 2^-56 + b 2^-84 + c 2^-112 (times the scales of the two vectors)
struct FxSum {
    long long a, b, c;
};

__device__ __forceinline__ void fx_zero(FxSum& s)
{
    s.a = s.b = s.c = 0;
}

__device__ __forceinline__ void fx_mad_wide(long long& s, int x, int y)
{
    asm("mad.wide.s32 %0, %1, %2, %0;" : "+l"(s) : "r"(x), "r"(y));
}

__device__ __forceinline__ void fx_mad(FxSum& s, const int4& x, const int4& y)
{
    fx_mad_wide(s.a, x.x, y.x);
    fx_mad_wide(s.b, x.x, y.y);
    fx_mad_wide(s.b, x.y, y.x);
    fx_mad_wide(s.c, x.x, y.z);
    fx_mad_wide(s.c, x.y, y.y);
    fx_mad_wide(s.c, x.z, y.x);
}

// a sum of at most three products as limbs again, at four times the product of its vectors' scales
__device__ __forceinline__ int4 fx_limbs(const FxSum& s)
{
    const long long d = (s.b + (s.c >> 28)) >> 2; // units of 2^-82
    const long long h = s.a + (d >> 26);          // units of 2^-56, |h| < 2^58
    const uint32_t d0 = static_cast<uint32_t>(d) & ((1u << 26) - 1u);
    return make_int4(static_cast<int>(h >> 30), static_cast<int>(static_cast<uint32_t>(h >> 2) & kFxMask),
                     static_cast<int>((static_cast<uint32_t>(h) & 3u) << 26 | d0), 0);
}

// the sum times 2^scale as a double (scale: sum of the vectors' unbiased scales), rounded to nearest
// (halves away from zero); the caller keeps the result inside the normal range
__device__ __forceinline__ double fx_to_double(const FxSum& s, int scale)
{
    const long long b = s.b + (s.c >> 28);
    long long h = s.a + (b >> 28); // value = (h 2^28 + l) 2^-84
    uint32_t l = static_cast<uint32_t>(b) & kFxMask;
    const uint32_t sign = h < 0 ? 0x80000000u : 0u;
    if (sign) {
        l = (0u - l) & kFxMask;
        h = ~h + (l == 0u ? 1 : 0);
    }
    if (h == 0) {
        if (l == 0u) return 0.0;
        h = l; // fewer than 28 bits: exact below
        l = 0u;
        scale -= 28;
    }
    const int lz = __clzll(h);
    const unsigned long long u =
        (static_cast<unsigned long long>(h) << lz) | (lz <= 28 ? static_cast<unsigned long long>(l >> (28 - lz))
                                                               : static_cast<unsigned long long>(l) << (lz - 28));
    // u in [2^63, 2^64): value = u 2^(28 - lz - 84 + scale)
    const unsigned long long m = ((u >> 1) + 0x200ull) >> 10; // 53 bits, or 2^53
    const int e = 1023 + 63 + 28 - lz - 84 + scale;
    return __longlong_as_double(static_cast<long long>((static_cast<unsigned long long>(e - 1) << 52) + m) |
                                static_cast<long long>(static_cast<unsigned long long>(sign) << 32));
}

} // namespace gfgpu
