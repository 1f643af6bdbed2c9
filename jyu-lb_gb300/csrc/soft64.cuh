// soft64.cuh -- correctly rounded FP64 operations on the integer pipes.
//
// GB300 issues one FP64 warp instruction per 19 cycles and SM, but two integer
// (ALU) warp instructions and two 32x32->64 multiply-adds per cycle.  An
// FP64 product with a constant takes 16 integer instructions and 4
// multiply-adds here (8 cycles), one addition of a chain of positive numbers
// in fixed point 11 (5.5 cycles), and both run beside the FP64 pipe.  Every
// function returns the bits that the IEEE operation with rounding to nearest
// even returns, on the operand ranges stated; callers check those ranges and
// take the plain operations otherwise.  The arithmetic follows IEEE 754 from
// its definition (exact product or sum, then one rounding) and runs on the
// host too, where the tests compare it with the hardware.
#pragma once
#include <stdint.h>
#include <string.h>

#include <cuda_runtime.h>

namespace jlb {
namespace soft64 {

#if defined(__CUDACC__)
#define S64_FN __host__ __device__ __forceinline__
#else
#define S64_FN inline
#endif

S64_FN uint64_t bits(double x) {
#ifdef __CUDA_ARCH__
    return (uint64_t)__double_as_longlong(x);
#else
    uint64_t u;
    memcpy(&u, &x, 8);
    return u;
#endif
}
S64_FN double from(uint32_t hi, uint32_t lo) {
#ifdef __CUDA_ARCH__
    return __hiloint2double((int)hi, (int)lo);
#else
    const uint64_t u = ((uint64_t)hi << 32) | lo;
    double x;
    memcpy(&x, &u, 8);
    return x;
#endif
}
// index of the highest set bit (of a nonzero word; 0xffffffff for 0)
S64_FN uint32_t top_bit(uint32_t x) {
#ifdef __CUDA_ARCH__
    uint32_t r;
    asm("bfind.u32 %0, %1;" : "=r"(r) : "r"(x));
    return r;
#else
    return x ? 31u - (uint32_t)__builtin_clz(x) : 0xffffffffu;
#endif
}
// the n low bits set, 0 <= n <= 31
S64_FN uint32_t low_mask(uint32_t n) {
#ifdef __CUDA_ARCH__
    uint32_t r;
    asm("bmsk.clamp.b32 %0, 0, %1;" : "=r"(r) : "r"(n));
    return r;
#else
    return (1u << n) - 1u;
#endif
}
// high word of (hi:lo) << s, 0 <= s <= 31
S64_FN uint32_t shl_hi(uint32_t lo, uint32_t hi, uint32_t s) {
#ifdef __CUDA_ARCH__
    return __funnelshift_l(lo, hi, s);
#else
    return s ? (hi << s) | (lo >> (32 - s)) : hi;
#endif
}
// low word of (hi:lo) >> s, 0 <= s <= 31
S64_FN uint32_t shr_lo(uint32_t lo, uint32_t hi, uint32_t s) {
#ifdef __CUDA_ARCH__
    return __funnelshift_r(lo, hi, s);
#else
    return s ? (lo >> s) | (hi << (32 - s)) : lo;
#endif
}

// A nonzero normal constant k prepared for mul(): its 53-bit significand
// shifted to [2^61, 2^62), and what its exponent and sign add to the high word
struct MulC {
    uint32_t hi, lo, base;
};
inline MulC make_mulc(double k) {
    const uint64_t u = bits(k);
    const uint64_t m = ((u & 0xfffffffffffffull) | (1ull << 52)) << 9;
    const uint32_t e = (uint32_t)(u >> 52) & 0x7ffu;
    return MulC{(uint32_t)(m >> 32), (uint32_t)m, ((e - 1024u) << 20) ^ (uint32_t)((u >> 63) << 31)};
}

// x * k for normal x with a normal product.  The 115-bit product's leading
// bits are shifted to 53; what is left out is one word with a sticky bit, into
// which the last kept bit goes too, so that "more than half" decides ties to
// even
S64_FN double mul(double x, const MulC &k) {
    const uint64_t u = bits(x);
    const uint32_t xh = (uint32_t)(u >> 32), l = (uint32_t)u;
    const uint32_t h = (xh & 0xfffffu) | 0x100000u;
    const uint64_t t0 = (uint64_t)l * k.lo;
    const uint64_t t1 = (uint64_t)h * k.lo + (t0 >> 32);
    const uint64_t t2 = (uint64_t)l * k.hi + t1;
    const uint64_t t3 = (uint64_t)h * k.hi + (t2 >> 32); // [2^49, 2^51)
    const uint32_t th = (uint32_t)(t3 >> 32), tl = (uint32_t)t3, w = (uint32_t)t2;
    const uint32_t c = th >> 18, s = 3u - c;
    const uint32_t ml = shl_hi(w, tl, s), mh = shl_hi(tl, th, s);
    const uint32_t low = (uint32_t)t0;
    const uint32_t sticky = low < 1u ? low : 1u;
    const uint32_t rest = (w << s) | ((sticky | ml) & 1u);
    const uint64_t up = ((uint64_t)rest + 0x7fffffffu) >> 32;
    const uint64_t m = (((uint64_t)mh << 32) | ml) + up;
    return from((uint32_t)(m >> 32) + (xh & 0xfff00000u) + k.base + (c << 20), (uint32_t)m);
}

// x * k for k > 0 where x may also be a zero (the product is then that zero);
// not for denormal x
S64_FN double mulz(double x, const MulC &k) {
    const double p = mul(x, k);
    const uint32_t xh = (uint32_t)(bits(x) >> 32);
    const bool zero = (xh & 0x7ff00000u) == 0u;
    return zero ? from(xh & 0x80000000u, 0u) : p;
}

// e + o and e - o for normal e > 0 and zero or normal o whose exponent is no
// larger: o is aligned to e's last place with 9 more bits and a sticky one
// (which only a shift by 10 or more sets), added and subtracted, and both results
// rounded, the smaller from at least 2^53 units of e's exponent - 61, that is
// 2^-8 of e's binade.  `least` collects the exponent difference (negative for a
// larger o); `close`, if given, the high word of the aligned difference, below
// 2^21 for a smaller or negative one.  |o| < e / 2 needs no such check.
S64_FN void add_sub(double e, double o, double &plus, double &minus, int32_t &least, int32_t *close = nullptr) {
    const uint64_t ue = bits(e), uo = bits(o);
    const uint32_t eh = (uint32_t)(ue >> 32), oh = (uint32_t)(uo >> 32);
    const uint32_t oe = (oh >> 20) & 0x7ffu;
    const int32_t r = (int32_t)(eh >> 20) - (int32_t)oe;
    least = least < r ? least : r;
    const uint64_t me = ((ue & 0xfffffffffffffull) | (1ull << 52)) << 9;
    const uint64_t mo = ((uo & 0xfffffffffffffull) | ((uint64_t)(oe < 1u ? oe : 1u) << 52)) << 9;
    const uint32_t sh = (uint32_t)r & 0x80000000u ? 0u : (uint32_t)r < 63u ? (uint32_t)r : 63u;
    const uint64_t v = mo >> sh;
    const uint64_t jam = v | ((v << sh) != mo ? 1u : 0u);
    if (close) {
        const int32_t q = (int32_t)(uint32_t)((me - jam) >> 32);
        *close = *close < q ? *close : q;
    }
    auto round = [&](uint64_t s) { // [2^53, 2^63)
        const uint32_t hi = (uint32_t)(s >> 32), lo = (uint32_t)s;
        const uint32_t d = (top_bit(hi) - 20u) & 31u;
        const uint32_t mask = low_mask(d), odd = (lo >> d) & 1u;
        s += (mask >> 1) + odd;
        return from(((uint32_t)(s >> 32) >> d) + ((eh & 0xfff00000u) + ((d - 10u) << 20)), shr_lo((uint32_t)s, (uint32_t)(s >> 32), d));
    };
    const double sum = round(me + jam), dif = round(me - jam);
    const bool neg = (oh >> 31) != 0u;
    plus = neg ? dif : sum;
    minus = neg ? sum : dif;
}

// ---------------------------------------------------------------------------
// Chains of additions in fixed point with unit 2^-61.  Each add() rounds as
// the FP64 addition does: to 53 significant bits of the partial sum.
// ---------------------------------------------------------------------------
constexpr uint32_t FIX_E0 = 1014; // exponent field of 2^-9, the least operand

// x in [2^-9, 2^(n-9)) as fixed point; `range` collects field - 1014, which is
// n or more for anything else (negative numbers, zeros, infinities, NaN)
S64_FN uint64_t fix(double x, uint32_t &range) {
    const uint64_t u = bits(x);
    const uint32_t xh = (uint32_t)(u >> 32), xl = (uint32_t)u;
    const uint32_t s = (xh >> 20) - FIX_E0;
    range = range > s ? range : s;
    const uint32_t h = (xh & 0xfffffu) | 0x100000u;
    return ((uint64_t)shl_hi(xl, h, s & 31u) << 32) | (uint32_t)(xl << (s & 31u));
}
// lo <= x < hi for positive bounds of at most 20 significant bits, by x's high
// word (false for negative numbers and NaN)
S64_FN bool within(double x, double lo, double hi) {
    const uint32_t l = (uint32_t)(bits(lo) >> 32), h = (uint32_t)(bits(hi) >> 32);
    return (uint32_t)(bits(x) >> 32) - l < h - l;
}

// a + b for positive operands (the sum is at least 2^53 units)
S64_FN uint64_t add(uint64_t a, uint64_t b) {
    const uint64_t s = a + b;
    const uint32_t hi = (uint32_t)(s >> 32), lo = (uint32_t)s;
    const uint32_t d = top_bit(hi) - 20u;
    const uint32_t mask = low_mask(d);
    const uint32_t odd = (lo >> d) & 1u;
    return (s + ((mask >> 1) + odd)) & ~(uint64_t)mask;
}
// a - b, expected positive and at least 2^53 units (checked through p; a
// negative difference has its top bit set, which the check sees as hi >= 2^31)
S64_FN uint64_t sub(uint64_t a, uint64_t b, uint32_t &p) {
    const uint64_t s = a - b;
    const uint32_t hi = (uint32_t)(s >> 32);
    const uint32_t q = hi - (1u << 21);
    p = p > q ? p : q; // below 2^31 - 2^21 for sums in range
    return add(s, 0);
}

// a fixed-point number already rounded to 53 bits, as a double
S64_FN double to_double(uint64_t s) {
    const uint32_t hi = (uint32_t)(s >> 32), lo = (uint32_t)s;
    const uint32_t d = top_bit(hi) - 20u;
    return from((hi >> d) + ((d + FIX_E0 - 1u) << 20), shr_lo(lo, hi, d));
}
// 1 / s for a fixed-point number rounded to 53 bits, as the correctly rounded
// double.  With s = D 2^d, D of 53 bits, it is q 2^(-44 - d) for the integer q
// nearest 2^105 / D: two Newton steps (x <- x + x (1 - D x)) from a 23-bit
// reciprocal give q to within one, and the remainder 2^105 - D q, below 2^54
// in size and so known from its low 64 bits, decides.  (No quotient lies
// midway: 2^106 / D would be an odd integer.)
S64_FN double recip(uint64_t s) {
    const uint32_t d = (top_bit((uint32_t)(s >> 32)) - 20u) & 31u;
    const uint64_t D = s >> d, dn = D << 11; // dn / 2^64 in [1/2, 1)
    const uint32_t dh = (uint32_t)(dn >> 32);
    // x0 / 2^30 = 2^64 / dn to about 2^-22, from the leading 24 bits
#ifdef __CUDA_ARCH__
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(__uint_as_float(0x3f000000u | ((dh >> 8) & 0x7fffffu))));
    const uint32_t x0 = (uint32_t)(y * 1073741824.0f);
#else
    const uint32_t x0 = (uint32_t)((1.0f / ((float)(dh >> 8) * 5.9604644775390625e-8f)) * 1073741824.0f);
#endif
    // e / 2^62 = 1 - dn x0 / 2^94, |e| < 2^42
    const uint64_t t = (uint64_t)dh * x0 + (((uint64_t)(uint32_t)dn * x0) >> 32);
    const int64_t e = (int64_t)((1ull << 62) - t);
    // x1 / 2^62, to about 2^-43
    const int64_t x1 = ((int64_t)x0 << 32) + (((e >> 12) * (int64_t)x0) >> 18);
    // the second step: e1 / 2^62 = 1 - dn x1 / 2^126, |e1| < 2^20
    const uint64_t xl = (uint32_t)x1, xh = (uint64_t)x1 >> 32;
    const uint64_t m1 = (uint64_t)dh * xl + (((uint64_t)(uint32_t)dn * xl) >> 32);
    const uint64_t m2 = (uint64_t)(uint32_t)dn * xh + (uint32_t)m1;
    const uint64_t p = (uint64_t)dh * xh + (m1 >> 32) + (m2 >> 32);
    const int64_t e1 = (int64_t)((1ull << 62) - p);
    const int64_t x2 = x1 + ((e1 * (int64_t)(x1 >> 32)) >> 30);
    uint64_t q = (uint64_t)(x2 + 512) >> 10; // x2 / 2^62 = 2^53 / D
    const int64_t rem = -(int64_t)(D * q);  // 2^105 - D q
    q += 2 * rem > (int64_t)D;
    q -= 2 * rem < -(int64_t)D;
    return from((uint32_t)(q >> 32) + ((1030u - d) << 20), (uint32_t)q);
}
// the signed difference a - b (|a - b| < 2^63 units) rounded to a double; an
// exact zero is +0 as in IEEE subtraction
S64_FN double diff_to_double(uint64_t a, uint64_t b) {
    const uint64_t s = a - b;
    const uint32_t sign = (uint32_t)(s >> 63);
    const uint64_t m = (s ^ (0ull - sign)) + sign;
    uint32_t hi = (uint32_t)(m >> 32), lo = (uint32_t)m, e = 1014u + 10u + 1u;
    // leading bit to bit 63
    if (hi == 0) { hi = lo; lo = 0; e -= 32u; }
    const uint32_t z = 31u - top_bit(hi); // 32 for zero
    const uint32_t nh = shl_hi(lo, hi, z & 31u), nl = lo << (z & 31u);
    // 53 of 64 bits stay
    const uint32_t ml = shr_lo(nl, nh, 11u), mh = nh >> 11;
    const uint32_t rest = (nl << 21) | (ml & 1u);
    const uint64_t up = ((uint64_t)rest + 0x7fffffffu) >> 32;
    const uint64_t r = (((uint64_t)mh << 32) | ml) + up;
    const uint32_t rh = (uint32_t)(r >> 32) + ((e - 1u - z) << 20) + (sign << 31);
    return hi == 0 ? 0.0 : from(rh, (uint32_t)r);
}

// ---------------------------------------------------------------------------
// Signed fixed-point products.  A 64-bit number is split into balanced 32-bit
// digits (low digit in [-2^31, 2^31)), so that three signed 32x32->64
// multiply-adds give the product's high half; the product of the two low
// digits, at most a quarter of the last place and zero on average, is left out.
// ---------------------------------------------------------------------------
struct Fix2 {
    int32_t hi, lo;
};
// -2^63 <= x < 2^63 - 2^31
S64_FN Fix2 digits(int64_t x) {
    Fix2 d;
    d.lo = (int32_t)(uint32_t)(uint64_t)x;
    d.hi = (int32_t)((x + 0x80000000ll) >> 32);
    return d;
}
// x y / 2^(64 - SH), rounded, for operands that digits() holds with
// |x| + |y| < 2^64 - 2^33 (the mixed products, below 2^31 (|x.hi| + |y.hi|) in
// size, and the rounding term then stay below 2^63) and a result of less than
// 2^63.  The collision's operands (lbm_fixed64.cuh), at most: 8 s 2^62 with the
// reciprocal 2^63 - 2^34; momenta and velocities 2^61.2; 9 (fe - y) + b and
// 6 fo - odd 2^62.6 with the rates 2^61.9; forces 2^60 with densities 2^61.6.
// Ties round up, with DOWN down.
template <int SH = 0, bool DOWN = false> S64_FN int64_t mulq(const Fix2 &x, const Fix2 &y) {
    int64_t m = (int64_t)x.lo * y.hi + ((0x80000000ll >> SH) - (DOWN ? 1 : 0));
    m = (int64_t)x.hi * y.lo + m;
    return (int64_t)x.hi * y.hi * (1ll << SH) + (m >> (32 - SH));
}
template <int SH = 0, bool DOWN = false> S64_FN int64_t mulq(int64_t x, const Fix2 &y) {
    return mulq<SH, DOWN>(digits(x), y);
}

// a positive number of 53 to 63 bits (unit 2^-61) rounded to a double;
// `low` collects what makes it 2^31 - 2^20 or more for any other number
S64_FN double round_to_double(int64_t v, uint32_t &low) {
    uint64_t s = (uint64_t)v;
    uint32_t hi = (uint32_t)(s >> 32);
    const uint32_t c = hi - (1u << 20);
    low = low > c ? low : c;
    const uint32_t d = (top_bit(hi) - 20u) & 31u;
    const uint32_t mask = low_mask(d), lo = (uint32_t)s;
    const uint32_t odd = (lo >> d) & mask & 1u;
    s = s + ((mask >> 1) + odd);
    hi = (uint32_t)(s >> 32);
    // bits below the last kept one go with the shift; a carry into the next
    // binade moves the exponent
    return from((hi >> d) + ((d + FIX_E0 - 1u) << 20), shr_lo((uint32_t)s, hi, d));
}
// a positive double in [2^-1, 2) with unit 2^-62
S64_FN int64_t fix62(double x) {
    const uint64_t u = bits(x);
    const uint32_t xh = (uint32_t)(u >> 32), xl = (uint32_t)u;
    const uint32_t s = ((xh >> 20) - (FIX_E0 - 1u)) & 31u;
    const uint32_t h = (xh & 0xfffffu) | 0x100000u;
    return (int64_t)(((uint64_t)shl_hi(xl, h, s) << 32) | (uint32_t)(xl << s));
}

} // namespace soft64
} // namespace jlb
