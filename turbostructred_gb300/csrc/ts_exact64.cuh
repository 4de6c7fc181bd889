// Correctly rounded FP64 division, square root and multiplication on the
// integer pipe.
//
// GB300 executes one FP64 warp instruction in 19 clocks per SM (76 per SM
// partition; measured), a division is 7.4 of them (141 clocks) and a square
// root 7.5 (143), while a 32x32->64 multiply-add takes 1.3 clocks and a plain
// integer operation 0.42.  The routines below form the same correctly
// rounded results (round to nearest even, so bit for bit those of `/` and
// sqrt()) in about 70 integer operations, and leave the FP64 pipe to the
// additions and multiplications.
//
// Method: Newton's iteration for the reciprocal (and the reciprocal square
// root) in fixed point from an FP32 seed, one second-order step (residual e
// of the seed, 1 + e + e^2 resp. 1 + e/2 + 3 e^2/8), then the integer
// quotient (root) n of 53 bits nearest to the fixed-point result and an exact
// integer remainder, a 2^k - n b resp. a 2^k - n^2, that says whether n or one
// of its neighbours is nearest.  Ties cannot occur: a quotient of two 53-bit
// integers, or a square root, that is a 54-bit odd integer would need an
// operand of more than 53 bits.
//
// Every normal operand is taken.  Zero divisors, subnormal operands and results,
// infinities and NaN are not: the routine reports them through `bad` and the
// caller takes the hardware operation instead.  A zero dividend, and a result
// that rounds to zero, are signed zeros.
//
// Compiles for the host too (the seed is then 1.0f / x, any seed within
// 2^-21 serves).
#pragma once

#include <cstdint>
#include <cstring>

#ifdef __CUDACC__
#define TS_X64 __host__ __device__ __forceinline__
#else
#include <cmath>
#define TS_X64 inline
#endif

namespace ts {
namespace x64 {

typedef uint32_t u32;
typedef uint64_t u64;
typedef int32_t i32;
typedef int64_t i64;

TS_X64 u64 bits_of(double d) {
#ifdef __CUDA_ARCH__
    return (u64)__double_as_longlong(d);
#else
    u64 b;
    std::memcpy(&b, &d, 8);
    return b;
#endif
}
TS_X64 double of_bits(u64 b) {
#ifdef __CUDA_ARCH__
    return __longlong_as_double((i64)b);
#else
    double d;
    std::memcpy(&d, &b, 8);
    return d;
#endif
}
TS_X64 u32 mulhi(u32 a, u32 b) {
#ifdef __CUDA_ARCH__
    return __umulhi(a, b);
#else
    return (u32)(((u64)a * b) >> 32);
#endif
}
// The words of a double.  Zero tests and magnitudes are formed on them: the
// compiler turns ((bits << 1) == 0) on the whole pattern back into a
// comparison on the FP64 pipe (seen as 19 clocks per test).
TS_X64 u32 hi_of(double d) {
#ifdef __CUDA_ARCH__
    return (u32)__double2hiint(d);
#else
    return (u32)(bits_of(d) >> 32);
#endif
}
TS_X64 u32 lo_of(double d) {
#ifdef __CUDA_ARCH__
    return (u32)__double2loint(d);
#else
    return (u32)bits_of(d);
#endif
}
TS_X64 double of_words(u32 hi, u32 lo) {
#ifdef __CUDA_ARCH__
    return __hiloint2double((i32)hi, (i32)lo);
#else
    return of_bits((u64)hi << 32 | lo);
#endif
}
TS_X64 bool is_zero(u32 hi, u32 lo) { return ((hi & 0x7FFFFFFFu) | lo) == 0u; }
TS_X64 u64 join(u32 hi, u32 lo) { return (u64)hi << 32 | lo; }
TS_X64 u64 wide(u32 a, u32 b) { return (u64)a * b; }

// FP32 seeds, biased down by 2^-21 (more than the seed's own error and that
// of its truncated argument) so that the Newton residual is positive, scaled
// to 30 fraction bits.
constexpr float kSeedScale = 1073741312.0f;  // 2^30 (1 - 2^-21)
TS_X64 u32 seed_rcp(u32 fbits) {
#ifdef __CUDA_ARCH__
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(__uint_as_float(fbits)));
    return __float2uint_rn(r * kSeedScale);
#else
    float f;
    std::memcpy(&f, &fbits, 4);
    return (u32)std::nearbyint((double)((1.0f / f) * kSeedScale));
#endif
}
TS_X64 u32 seed_rsqrt(u32 fbits) {
#ifdef __CUDA_ARCH__
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(__uint_as_float(fbits)));
    return __float2uint_rn(r * kSeedScale);
#else
    float f;
    std::memcpy(&f, &fbits, 4);
    return (u32)std::nearbyint((double)((float)(1.0 / std::sqrt((double)f)) * kSeedScale));
#endif
}

// A divisor prepared once for any number of quotients: its 53-bit
// significand B and Y = 2^114 / B to a few units.
struct Divisor {
    u64 B, Y;
    int e;
    u32 sign;
};

// b: normal, else `bad`.
TS_X64 Divisor divisor(double b, bool& bad) {
    const u32 hi = hi_of(b);
    const u32 e = (hi >> 20) & 0x7FFu;
    bad |= e - 1u >= 2046u;
    Divisor d;
    d.e = (int)e;
    d.sign = hi & 0x80000000u;
    d.B = join((hi & 0xFFFFFu) | 0x100000u, lo_of(b));
    const u64 bs = d.B << 11;  // significand in [1, 2) with 63 fraction bits
    const u32 bh = (u32)(bs >> 32), bl = (u32)bs;
    const u32 r = seed_rcp(0x3F800000u | ((bh >> 8) & 0x7FFFFFu));
    // residual 1 - b r with 61 fraction bits: 0 < E < 2^41
    const u64 E = (1ull << 61) - (wide(bh, r) + mulhi(bl, r));
    const u32 eh = (u32)(E >> 20);
    const u64 T = E + (wide(eh, eh) >> 21);  // E + E^2
    const u32 th = (u32)(T >> 32), tl = (u32)T;
    d.Y = ((u64)r << 32) + (wide(r, th) << 3) + (wide(r, tl) >> 29);
    return d;
}

// RN(a / b).  a: zero or normal, with a quotient that is normal or rounds to
// zero; else `bad`.
TS_X64 double quotient(double a, const Divisor& d, bool& bad) {
    const u32 ahi = hi_of(a), alo = lo_of(a);
    const u32 sign = (ahi ^ d.sign) & 0x80000000u;
    const u32 e = (ahi >> 20) & 0x7FFu;
    u64 A = join((ahi & 0xFFFFFu) | 0x100000u, alo);
    const u32 lt = A < d.B ? 1u : 0u;
    A <<= lt;  // in [B, 2B): the quotient's significand is in [2^52, 2^53]
    const u64 aq = A << 9;
    const u32 qh = (u32)(aq >> 32), ql = (u32)aq;
    const u32 yh = (u32)(d.Y >> 32), yl = (u32)d.Y;
    const u64 h = wide(qh, yh) + mulhi(qh, yl) + mulhi(ql, yh);  // quotient with 7 extra bits
    u64 n = (h + 64) >> 7;
    // exact remainder of the candidate (|R| < 2^53: the low 64 bits hold it)
    const u64 R2 = ((A << 52) - n * d.B) << 1;
    n += (d.B - R2) >> 63;  // 2R > B: the next one is nearer
    n -= (d.B + R2) >> 63;  // 2R < -B: the previous one
    const bool none = is_zero(ahi, alo);
    const int E = (int)e - d.e + 1023 - (int)lt;  // (one more where n = 2^53: E = 0 counts as subnormal)
    const bool zero = none || E < -52;  // less than half the smallest subnormal
    bad |= !((e - 1u < 2046u || none) && ((u32)(E - 1) < 2046u || zero));
    const u32 qhi = (u32)(n >> 32) + ((u32)(E - 1) << 20);
    return of_words((zero ? 0u : qhi) | sign, zero ? 0u : (u32)n);
}

TS_X64 double div(double a, double b, bool& bad) { return quotient(a, divisor(b, bad), bad); }

// RN(sqrt(a)).  a: positive and normal, else `bad`.
TS_X64 double root(double a, bool& bad) {
    const u32 hi = hi_of(a), lo = lo_of(a);
    const u32 e = hi >> 20;  // with the sign: negative numbers are out of range too
    bad |= e - 1u >= 2046u;
    const u32 odd = (e & 1u) ^ 1u;  // a = m 2^(2k), m in [1, 4)
    const u64 M = join((hi & 0xFFFFFu) | 0x100000u, lo) << odd;
    const u64 ms = M << 9;  // m with 61 fraction bits
    const u32 mh = (u32)(ms >> 32), ml = (u32)ms;
    const u32 r = seed_rsqrt(((127u + odd) << 23) | ((hi & 0xFFFFFu) << 3) | (lo >> 29));
    const u64 G = wide(mh, r) + mulhi(ml, r);  // m r ~ sqrt(m), 59 fraction bits
    const u32 gh = (u32)(G >> 32), gl = (u32)G;
    const u64 E = (1ull << 57) - (wide(gh, r) + mulhi(gl, r));  // 1 - m r^2, 57 fraction bits, 0 < E < 2^38
    const u32 eh = (u32)(E >> 16);
    const u64 C = E + ((3 * wide(eh, eh)) >> 27);  // E + 3/4 E^2
    const u32 ch = (u32)(C >> 32), cl = (u32)C;
    // G C / 2^38 (without the lowest partial product), then / 2^58
    const u64 W = (wide(gh, cl) >> 6) + (wide(gh, ch) << 26) + ((mulhi(gl, cl) + wide(gl, ch)) >> 6);
    const u64 S = G + (W >> 20);
    u64 n = (S + 64) >> 7;
    // exact remainder of the candidate: n is nearest iff -n < R <= n
    const u64 R = (M << 52) - n * n;
    const u64 up = (n - R) >> 63, down = (n + R - 1) >> 63;
    n = n + up - down;
    const int k = ((int)e - 1023 - (int)odd) >> 1;
    return of_words((u32)(n >> 32) + ((u32)(k + 1022) << 20), (u32)n);
}

// RN(a b).  a and b: zero or normal, with a product that is normal or rounds to
// zero; else `rare` (nothing is wrong then: the caller lets the hardware multiply).  The exact
// 106-bit product in four 32x32->64 multiply-adds, one bit of normalisation,
// and the rounding carry added through the exponent: about 30 plain integer
// operations, 12 to 14 clocks per warp and SM beside the FP64 pipe's 19.
TS_X64 double mul(double a, double b, bool& rare) {
    const u32 ahi = hi_of(a), al = lo_of(a), bhi = hi_of(b), blo = lo_of(b);
    const u32 ea = ahi & 0x7FF00000u, eb = bhi & 0x7FF00000u;  // exponents in place
    const bool za = is_zero(ahi, al), zb = is_zero(bhi, blo);
    const u32 ah = (ahi & 0xFFFFFu) | 0x100000u;
    const u64 B = join((bhi & 0xFFFFFu) | 0x100000u, blo) << 10;  // 63 bits
    const u32 bh = (u32)(B >> 32), bl = (u32)B;
    const u64 p0 = wide(al, bl);
    const u64 p1 = wide(ah, bl) + (u32)(p0 >> 32);
    const u64 p2 = wide(al, bh) + p1;  // < 2^63 + 2^54
    const u64 p3 = wide(ah, bh) + (u32)(p2 >> 32);
    // product = p3 2^64 + lo(p2) 2^32 + lo(p0), in [2^114, 2^116)
    const u32 ph = (u32)(p3 >> 32), pm = (u32)p3, pl = (u32)p2;
    const u32 top = ph >> 19;  // 1: 2^115 or more
    const u32 s = 2u - top;
    // 53 bits nh:nl, the rest in r (its lowest bit: anything below)
    u32 nh = (ph << s) | (pm >> (32 - s)), nl = (pm << s) | (pl >> (32 - s));
    const u32 r = (pl << s) | ((u32)p0 != 0u ? 1u : 0u);
    // carry out of r + 0x7FFFFFFF + (nl & 1): above one half, or a tie and nl odd
    const u32 half_up = 0x7FFFFFFFu + (nl & 1u);
    const u32 es = ea + eb + (top << 20);  // the biased exponent + 1023: no carry out
    const u32 e = es - (1024u << 20);      // with the leading bit of nh
    const bool zero = za || zb || es < (971u << 20);  // less than half the smallest subnormal
    rare = !((ea - (1u << 20) < (2046u << 20) || za) && (eb - (1u << 20) < (2046u << 20) || zb) &&
             (e < (2046u << 20) || zero));
#ifdef __CUDA_ARCH__
    u32 drop;
    asm("add.cc.u32 %0, %3, %4;\n\taddc.cc.u32 %1, %1, 0;\n\taddc.u32 %2, %2, %5;"
        : "=r"(drop), "+r"(nl), "+r"(nh)
        : "r"(r), "r"(half_up), "r"(e));
#else
    const u32 c = (u32)(((u64)r + half_up) >> 32);
    const u64 n = join(nh, nl) + c;
    nh = (u32)(n >> 32) + e;
    nl = (u32)n;
#endif
    return of_words((zero ? 0u : nh) | ((ahi ^ bhi) & 0x80000000u), zero ? 0u : nl);
}

// x / 2 (exact): zero or a normal number whose half is normal, else `bad`.
TS_X64 double half(double x, bool& bad) {
    const u32 hi = hi_of(x), lo = lo_of(x);
    const u32 e = (hi >> 20) & 0x7FFu;
    const bool zero = is_zero(hi, lo);
    bad |= !(zero || e - 2u < 2045u);
    return of_words(zero ? hi : hi - 0x00100000u, lo);
}

}  // namespace x64
}  // namespace ts
