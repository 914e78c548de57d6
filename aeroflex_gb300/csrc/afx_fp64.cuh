// IEEE-754 double-precision division, square root and ordering in integer
// arithmetic.
//
// Why: an SM of sm_103a has two FP64 lanes and 128 lanes for 32-bit integer
// and FP32 work, so one FP64 instruction of a warp holds the FP64 pipe for
// as long as the four schedulers need to issue some sixty integer ones.  A
// double division is a chain of FP64 instructions; here it is about fifty
// integer instructions and none on the FP64 pipe.  The FP64 kernels of this
// library are bound by that pipe, so divisions, square roots and compares
// are moved off it; additions and products stay on it.
//
// Results are those of IEEE-754 round-to-nearest-even, bit for bit:
//   * a quotient of two significands X, Y (53-bit integers) is formed as the
//     integer floor(X 2^53 / Y) by two steps of long division with a 32-bit
//     reciprocal of Y that is never too large, exact 64-bit remainders and a
//     final correction.  A quotient of two 53-bit numbers is never half way
//     between two 53-bit numbers, so adding half a unit to the 54-bit floor
//     rounds it correctly;
//   * a square root likewise from floor(sqrt(V 2^106)), by two steps with a
//     32-bit reciprocal square root (never half way either);
//   * operands that are zero, subnormal, infinite or NaN, and results outside
//     the normal range, take the compiler's own division, square root or
//     product (a zero over a normal number, and a zero times a finite one, are
//     answered here).
// The reciprocal seeds are the hardware's single-precision approximations
// (3 ulp allowed for) and one Newton step in 32-bit fixed point.
#pragma once

#include <cstdint>

#ifdef __CUDACC__
#define AFX_HD __host__ __device__ __forceinline__
#else
#define AFX_HD inline
#endif

namespace afx {
namespace fp64 {

// ---- machine access; the host forms let the algorithms be tested without a GPU
AFX_HD uint64_t bits_of(const double x) {
#ifdef __CUDA_ARCH__
    // two words by hand: the compiler turns integer tests of a reinterpreted
    // double (such as "is zero") back into compares on the FP64 pipe
    uint32_t lo, hi;
    asm("mov.b64 {%0, %1}, %2;" : "=r"(lo), "=r"(hi) : "d"(x));
    return ((uint64_t)hi << 32) | lo;
#else
    uint64_t u;
    __builtin_memcpy(&u, &x, 8);
    return u;
#endif
}
AFX_HD double of_bits(const uint64_t u) {
#ifdef __CUDA_ARCH__
    return __longlong_as_double((long long)u);
#else
    double x;
    __builtin_memcpy(&x, &u, 8);
    return x;
#endif
}
AFX_HD uint32_t mulhi(const uint32_t a, const uint32_t b) {
#ifdef __CUDA_ARCH__
    return __umulhi(a, b);
#else
    return (uint32_t)(((uint64_t)a * b) >> 32);
#endif
}
AFX_HD int32_t mulhi_s(const int32_t a, const int32_t b) {
#ifdef __CUDA_ARCH__
    return __mulhi(a, b);
#else
    return (int32_t)(((int64_t)a * b) >> 32);
#endif
}
#ifndef __CUDA_ARCH__
extern int seed_ulps;  // host tests: error added to the seeds, in units of their last place
inline float f32_of(const uint32_t u) { float f; __builtin_memcpy(&f, &u, 4); return f; }
inline uint32_t f32_bits(const float f) { uint32_t u; __builtin_memcpy(&u, &f, 4); return u; }
#endif
// approximate 1/f and 1/sqrt(f) of the float with bits u, as bits, kept in [0.5, 1)
AFX_HD uint32_t seed_rcp(const uint32_t u) {
#ifdef __CUDA_ARCH__
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(__uint_as_float(u)));
    return __float_as_uint(fminf(fmaxf(r, 0.5f), 0.99999994f));
#else
    const uint32_t r = f32_bits(1.0f / f32_of(u)) + (uint32_t)seed_ulps;
    return r < 0x3f000000u ? 0x3f000000u : (r > 0x3f7fffffu ? 0x3f7fffffu : r);
#endif
}
AFX_HD uint32_t seed_rsqrt(const uint32_t u) {
#ifdef __CUDA_ARCH__
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(__uint_as_float(u)));
    return __float_as_uint(fminf(fmaxf(r, 0.5f), 0.99999994f));
#else
    const uint32_t r = f32_bits((float)(1.0 / __builtin_sqrt((double)f32_of(u)))) + (uint32_t)seed_ulps;
    return r < 0x3f000000u ? 0x3f000000u : (r > 0x3f7fffffu ? 0x3f7fffffu : r);
#endif
}

// The compiler's own operations for the rare operands: out of line, so that
// the paths around them stay short and are branched over.
#ifdef __CUDACC__
#define AFX_RARE static __host__ __device__ __noinline__
#define AFX_RARE_CALL (void)0
#else
#define AFX_RARE static
inline long rare_calls = 0;  // host tests: operands that got here
#define AFX_RARE_CALL (void)++rare_calls
#endif
AFX_RARE double div_rare(const double x, const double y) {
    AFX_RARE_CALL;
    return x / y;
}
AFX_RARE double root_rare(const double x) {
    AFX_RARE_CALL;
#ifdef __CUDACC__
    return sqrt(x);
#else
    return __builtin_sqrt(x);
#endif
}
// What mul() does not form itself.  A zero times a finite number is common (a
// uniform stream has no differences, a level one no cross flow) and is answered
// off the FP64 pipe: 1.05M cells of uniform stream, five iterations, 15.45 ->
// 14.51 ms, a disturbed stream the same.  (In mul() itself the test cost the
// disturbed one 3 to 4%.)
AFX_RARE double mul_rare(const double x, const double y) {
    const uint64_t u = bits_of(x), v = bits_of(y);
    const uint64_t inf = 0xffe0000000000000ull;  // shifted past the sign
    if ((u << 1 == 0ull && v << 1 < inf) || (v << 1 == 0ull && u << 1 < inf))
        return of_bits((u ^ v) & 0x8000000000000000ull);
    AFX_RARE_CALL;
    return x * y;
}

// (double)x, FP32 subnormals as zero (as the FP32 kernels are compiled)
AFX_HD double widen(const uint32_t u) {
    const uint32_t e = (u >> 23) & 0xffu, mag = u & 0x7fffffffu;
    const uint32_t hi = (mag >> 3) + (e == 0xffu ? 0x70000000u : 0x38000000u);
    const uint64_t v = e == 0 ? 0ull : ((uint64_t)hi << 32) | (u << 29);
    return of_bits(v | ((uint64_t)(u & 0x80000000u) << 32));
}
// bits of (float)x, round to nearest even; false outside FP32's normal range
// (other than zero)
AFX_HD bool narrow(const double x, uint32_t& r) {
    const uint64_t u = bits_of(x);
    const uint32_t hi = (uint32_t)(u >> 32), lo = (uint32_t)u, sgn = hi & 0x80000000u;
    const uint32_t e = (hi >> 20) & 0x7ffu;
    const uint32_t m = ((e - 896u) << 23) | ((hi & 0xfffffu) << 3) | (lo >> 29);
    const uint32_t rem = lo & 0x1fffffffu;
    r = (m + (rem + (m & 1u) > 0x10000000u ? 1u : 0u)) | sgn;
    if ((hi << 1 | lo) == 0u) r = sgn;
    return e - 897u < 254u || (hi << 1 | lo) == 0u;
}

// A denominator: its significand and a 32-bit reciprocal, shared by the
// quotients that divide by it.
struct Den {
    double y;
    uint64_t Y;    // significand, 2^52 <= Y < 2^53
    uint32_t r;    // 2^84 / Y - 8 < r <= 2^84 / Y
    int32_t e;     // biased exponent
    uint32_t sgn;  // sign bit
};

AFX_HD Den den(const double y) {
    Den d;
    const uint64_t u = bits_of(y);
    const uint32_t hi = (uint32_t)(u >> 32);
    d.y = y;
    d.sgn = hi & 0x80000000u;
    d.e = (int32_t)((hi >> 20) & 0x7ffu);
    d.Y = (u & 0x000fffffffffffffull) | 0x0010000000000000ull;
    const uint32_t Y32 = (uint32_t)(d.Y >> 21);  // [2^31, 2^32)
    // 1/y from the next float above the leading 24 bits: in [0.5, 1)
    const uint32_t s = seed_rcp(0x3f800001u + ((Y32 >> 8) & 0x7fffffu));
    const uint32_t r0 = (s << 8) | 0x80000000u;  // its significand, in units of 2^-32
    // one Newton step: r0 + r0 (1 - y r0), the residual in units of 2^-63
    const int64_t err = (int64_t)(0x8000000000000000ull - (uint64_t)Y32 * r0);
    // less 3: the leading bits of y alone can make the reciprocal 2 units too large
    d.r = r0 - 3u + (uint32_t)(mulhi_s((int32_t)(r0 >> 1), (int32_t)(err >> 11)) >> 19);
    return d;
}

// the denominator 2 y
AFX_HD Den twice(const Den& a) {
    Den d = a;
    const bool plain = (uint32_t)(a.e - 1) < 2045u;
    d.y = plain ? of_bits(bits_of(a.y) + 0x0010000000000000ull) : a.y + a.y;
    d.e = plain ? a.e + 1 : 0;  // 0: not for the integer path
    return d;
}

// x / d
AFX_HD double quot(const double x, const Den& d) {
    const uint64_t u = bits_of(x);
    const uint32_t hi = (uint32_t)(u >> 32);
    const int32_t ex = (int32_t)((hi >> 20) & 0x7ffu);
    const uint64_t X = (u & 0x000fffffffffffffull) | 0x0010000000000000ull;
    // quotient in [1, 2): R = X - Y, or 2 X - Y one binade lower
    uint64_t R = X - d.Y;
    const bool low = (int64_t)R < 0;
    R += low ? X : 0ull;
    const int32_t e = ex - d.e + (low ? 1022 : 1023);
    // 31 quotient bits (at most 8 too small), then 22 more (at most 1 too small)
    const uint32_t d1 = mulhi((uint32_t)(R >> 21), d.r);
    R = (R << 31) - (uint64_t)d1 * d.Y;  // [0, 9 Y)
    const uint32_t d2 = mulhi((uint32_t)(R >> 25), d.r) >> 5;
    R = (R << 22) - (uint64_t)d2 * d.Y;  // [0, 2 Y)
    const uint64_t Q = 0x0020000000000000ull + ((uint64_t)d1 << 22) + d2 + (R >= d.Y ? 2u : 1u);
    const uint32_t sgn = (hi ^ d.sgn) & 0x80000000u;
    uint64_t q = ((uint64_t)((uint32_t)((e - 1) << 20) | sgn) << 32) + (Q >> 1);
    const bool y_ok = (uint32_t)(d.e - 1) < 2046u;
    const bool zero = (u << 1) == 0ull;
    if (zero) q = (uint64_t)sgn << 32;
    if (y_ok && (zero || ((uint32_t)(ex - 1) < 2046u && (uint32_t)(e - 1) < 2046u))) return of_bits(q);
    return div_rare(x, d.y);
}

AFX_HD double div(const double x, const double y) { return quot(x, den(y)); }

AFX_HD double root(const double x) {
    const uint64_t u = bits_of(x);
    const int32_t e = (int32_t)(u >> 52);  // sign included: a negative number is out of range below
    const bool odd = (e & 1) == 0;         // bias 1023: an even biased exponent is an odd power of two
    uint64_t W = (u & 0x000fffffffffffffull) | 0x0010000000000000ull;  // v = W 2^-52
    if (odd) W <<= 1;                                                  // v in [1, 4)
    const uint32_t V32 = (uint32_t)(W >> 22);                          // [2^30, 2^32)
    // 1/sqrt(v) from the next float above the leading bits: in [0.5, 1)
    const uint32_t lead = (uint32_t)(u >> 29) & 0x7fffffu;
    const uint32_t s = seed_rsqrt((odd ? 0x40000001u : 0x3f800001u) + lead);
    const uint32_t y0 = (s << 8) | 0x80000000u;  // units of 2^-32
    // one Newton step: y0 + y0 (1 - v y0^2) / 2, the residual in units of 2^-62
    const int64_t err = (int64_t)(0x4000000000000000ull - (uint64_t)V32 * mulhi(y0, y0));
    const uint32_t y = y0 - 8u + (uint32_t)(mulhi_s((int32_t)(y0 >> 1), (int32_t)(err >> 11)) >> 19);
    // 31 bits of the root (a little too small), remainder, 23 more
    const uint32_t d1 = mulhi(V32, y);
    const uint64_t R1 = (W << 8) - (uint64_t)d1 * d1;
    const int32_t d2 = (int32_t)(mulhi((uint32_t)(R1 >> 4), y) >> 4) - 1;
    uint64_t S = ((uint64_t)d1 << 23) + (uint64_t)(int64_t)d2;
    int64_t R = (int64_t)((R1 << 46) - ((uint64_t)((int64_t)d1 * d2) << 24) - (uint64_t)((int64_t)d2 * d2));
    // S is the floor or up to two below it
    int64_t t = R - (int64_t)(2 * S + 1);
    if (t >= 0) {
        R = t;
        S += 1;
    }
    t = R - (int64_t)(2 * S + 1);
    if (t >= 0) S += 1;
    const uint64_t q = ((uint64_t)(uint32_t)(((e + 1023) >> 1) - 1) << 52) + ((S + 1) >> 1);
    if ((uint32_t)(e - 1) < 2046u) return of_bits(q);
    return root_rare(x);
}

// x y.  The FP64 pipe does this in one instruction that holds it for 18.6 cycles;
// this takes some forty integer instructions beside it.  Kernels that the pipe
// bounds give a share of their products to the integer lanes (see roe_flux2).
AFX_HD double mul(const double x, const double y) {
    const uint64_t u = bits_of(x), v = bits_of(y);
    const uint32_t ah = (uint32_t)(u >> 32), bh = (uint32_t)(v >> 32), al = (uint32_t)u, bl = (uint32_t)v;
    const uint32_t ea = (ah >> 20) & 0x7ffu, eb = (bh >> 20) & 0x7ffu;
    // 53-bit significand times 53 bits moved up by 11: the upper word of the
    // 128-bit product holds the leading 52 or 53 bits
    const uint32_t Ah = (ah & 0xfffffu) | 0x100000u;
    const uint32_t Bh = ((bh << 11) | (bl >> 21)) | 0x80000000u, Bl = bl << 11;
    const uint64_t p00 = (uint64_t)al * Bl;
    const uint64_t p01 = (uint64_t)al * Bh + (uint32_t)(p00 >> 32);
    const uint64_t p10 = (uint64_t)Ah * Bl + (uint32_t)p01;
    uint64_t hi = (uint64_t)Ah * Bh + (uint32_t)(p01 >> 32) + (uint32_t)(p10 >> 32);
    uint32_t fr = (uint32_t)p10;           // the next 32 bits
    const uint32_t rest = (uint32_t)p00;   // and the last ones
    const bool low = (uint32_t)(hi >> 32) < 0x100000u;
    if (low) {
        hi = (hi << 1) | (fr >> 31);
        fr = (fr << 1) | (rest >> 31);
    }
    // half a unit or more, a tie to even
    const uint32_t tie = (rest | ((uint32_t)hi & 1u)) == 0u ? 1u : 0u;
    hi += fr > 0x7fffffffu + tie ? 1u : 0u;
    const int32_t e = (int32_t)(ea + eb) - (low ? 1023 : 1022);
    const uint32_t top = ((uint32_t)(e - 1) << 20) | ((ah ^ bh) & 0x80000000u);
    if (ea - 1u < 2046u && eb - 1u < 2046u && (uint32_t)(e - 1) < 2046u) return of_bits(((uint64_t)top << 32) + hi);
    return mul_rare(x, y);
}

// two's complement order of the sign-magnitude numbers (-0 counts as +0)
AFX_HD int64_t order_of(const double x) {
    const int64_t i = (int64_t)bits_of(x);
    return i < 0 ? (int64_t)(0x8000000000000000ull - (uint64_t)i) : i;
}
// a < b and a <= b; a NaN is beyond an infinity, so the two limits make any
// comparison with one false
AFX_HD bool less(const double a, const double b) {
    const int64_t i = order_of(a), j = order_of(b), inf = 0x7ff0000000000000ll;
    return i < j && i >= -inf && j <= inf;
}
AFX_HD bool less_equal(const double a, const double b) {
    const int64_t i = order_of(a), j = order_of(b), inf = 0x7ff0000000000000ll;
    return i <= j && i >= -inf && j <= inf;
}

}  // namespace fp64
}  // namespace afx
