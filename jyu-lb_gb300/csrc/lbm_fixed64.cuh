// lbm_fixed64.cuh -- BGK / TRT / regularized collision in 64-bit fixed point,
// for populations stored in FP64 (precision JLB_FP64_FAST).
//
// GB300's FP64 pipe bounds an FP64 collision at 19 cycles per warp
// instruction and SM, where a 64-bit integer addition takes one cycle and a
// signed 64-bit high product three multiply-adds.  In fixed point with unit
// 2^-61 the populations are exact (they are doubles of at least 2^-9), every
// sum is exact, and a product rounds at 2^-62, where a double of a population's
// size rounds at 2^-58 or above: the collision loses less than FP64 arithmetic
// does, and only the store rounds to 53 bits.  One FP64 reciprocal is left, for
// the FP64 pipe has nothing else to do (soft64.cuh's: 128^3 145 -> 169 us a step).
//
// With pairs (m, p) of opposite populations, even part fe = f_p + f_m, odd
// part fo = f_p - f_m, weight w and direction c of p, the update
// (jyulb/D3Q19.pyx:655-853) is f_p - E - O, f_m - E + O with
//   E = we/2 fe - w (we den + 4.5 cc:H2 - 1.5 tr H2)
//     = we/72 (36 fe - 36 w (2 den - 3 tr S + 9 cc:S)),
//   O = wo/2 fo - 3 w c.(wo s + c1 a den) = wo/12 (6 fo - 36 w c.(j + a den / wo)),
// where s = j + a den/2 = den u, c1 = 1 - wo/2 and
//   S = s u + (c2/we) (a s + s a), c2 = 1 - we/2;
// the rest population takes what the pairs give (their sum is conserved
// exactly).  The regularized update (jyulb/D3Q19.pyx:859-940) projects
//   H1 = j + a den, H2 = P + we (S - P), P = sum c c f - den/3.
#pragma once
#include <cmath>

#include "soft64.cuh"

namespace jlb {

// constants of the fixed-point collision, formed by the host
struct FixConsts {
    soft64::Fix2 e, o;     // we/72 (2^66), wo/12 (2^64)
    soft64::Fix2 w;        // we (2^61), regularized
    soft64::Fix2 c72, c12; // 1/72 (2^68), 1/12 (2^64), regularized
    soft64::Fix2 ah[3];    // a/2 (2^64)
    soft64::Fix2 ao[3];    // a/wo (2^64); regularized: a
    soft64::Fix2 k2[3];    // (c2/we) a (2^62)
    int64_t k[3];          // the same as a number
    unsigned mask;         // components of a that are not zero
    int ok;                // rates and force within the form's range
};

inline int64_t fix_round(double x, int m) { return (int64_t)std::llrint(std::ldexp(x, m)); }
inline int64_t fix_unit(int m, int n) { // 2^m / n, rounded
    return (int64_t)(((((unsigned __int128)1 << (m + 1)) / (unsigned)n) + 1) >> 1);
}
inline FixConsts make_fix_consts(bool trt, bool reg, double we, double wo, const double g[3]) {
    FixConsts k{};
    if (!trt) wo = we;
    const double c2w = (1.0 - 0.5 * we) / we;
    k.ok = we > 0.0 && we < 2.0 && wo > 0.0 && wo < 2.0;
    for (int d = 0; d < 3; ++d) {
        const double ao = reg ? g[d] : g[d] / wo;
        if (g[d] != 0.0) k.mask |= 1u << d;
        if (!(std::fabs(g[d]) < 0x1p-4 && std::fabs(ao) < 0x1p-4 && std::fabs(c2w * g[d]) < 0x1p-4)) k.ok = 0;
    }
    if (!k.ok) return k;
    k.e = soft64::digits(fix_round(we / 72.0, 66));
    k.o = soft64::digits(fix_round(wo / 12.0, 64));
    k.w = soft64::digits(fix_round(we, 61));
    k.c72 = soft64::digits(fix_unit(68, 72));
    k.c12 = soft64::digits(fix_unit(64, 12));
    for (int d = 0; d < 3; ++d) {
        k.ah[d] = soft64::digits(fix_round(0.5 * g[d], 64));
        k.ao[d] = soft64::digits(fix_round(reg ? g[d] : g[d] / wo, 64));
        k.k[d] = fix_round(c2w * g[d], 62);
        k.k2[d] = soft64::digits(k.k[d]);
    }
    return k;
}

// What the density's range leaves the rest population, near equilibrium.  Looked
// at before anything else, so that a site with a density not near 1 pays for
// nothing but the FP64 form.
S64_FN bool fixed_range(const double *f) { return soft64::within(f[9], 0.125, 0.5); }

// f[19] in place; returns false where an operand leaves the form's range:
// populations in [2^-9, 1/8) (rest: fixed_range()) before and at least 2^-9
// after, density in [1/2 + 2^-29, 3/2), |j + a den/2| < 1/4 per component; f is then undefined.
// (From density 1/2 itself the reciprocal, with unit 2^-62, would reach 2^63: the
// margin leaves digits() the 2^31 it adds.)  With `want`, mom receives den and
// the stored velocity u = j/den + a/2.
//
// The products that relax the even and odd parts round ties up, with DOWN down,
// and the steps of the AA pair take turns.  A rate such as wo/12 = 1/16 (tau 0.8,
// magic 1/4) makes a tie of every 16th product, and rounding all of them up
// moved the momentum by 8e-19 a step and site, always the same way; FP64's own
// bias is 1e-20 to 1e-19.
template <bool REG, bool DOWN = false>
S64_FN bool collide_fixed(double *f, const FixConsts &k, const double *a, bool want, double *mom) {
    using namespace soft64;
    if (!fixed_range(f)) return false;
    uint32_t range = 0, rest = 0;
    int64_t x[19];
#pragma unroll
    for (int q = 0; q < 19; ++q) x[q] = (int64_t)fix(f[q], q == 9 ? rest : range);
    // even and odd parts of the pairs, by the index of their p: 10 (0,0,1),
    // 11 (0,1,-1), 12 (0,1,0), 13 (0,1,1), 14 (1,-1,0), 15 (1,0,-1),
    // 16 (1,0,0), 17 (1,0,1), 18 (1,1,0)
    int64_t fe[9], fo[9]; // [p - 10]
#pragma unroll
    for (int i = 0; i < 9; ++i) {
        fe[i] = x[10 + i] + x[8 - i];
        fo[i] = x[10 + i] - x[8 - i];
    }
    const int64_t den = ((fe[0] + fe[1]) + (fe[2] + fe[3])) + ((fe[4] + fe[5]) + (fe[6] + fe[7])) + (fe[8] + x[9]);
    const int64_t j[3] = {((fo[4] + fo[5]) + (fo[6] + fo[7])) + fo[8], ((fo[1] + fo[2]) + (fo[3] - fo[4])) + fo[8],
                          ((fo[0] - fo[1]) + (fo[3] - fo[5])) + fo[7]};
    uint32_t unused = 0;
    const double dd = round_to_double(den, unused);
    const double inv = 1.0 / dd;
    const Fix2 iv = digits(fix62(inv));
    int64_t s[3], u[3]; // momentum (2^61) and velocity (2^62) of the step's middle
    uint32_t fast = 0;
    Fix2 sd[3];
    Fix2 dn = digits(den);
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        s[d] = j[d];
        if ((k.mask >> d) & 1u) s[d] += mulq(dn, k.ah[d]);
        const uint32_t r = (uint32_t)((uint64_t)s[d] >> 32) + (1u << 27);
        fast = fast > r ? fast : r;
        u[d] = mulq(s[d] * 8, iv);
        sd[d] = digits(s[d]);
    }
    if (range > 5u || fast >= (1u << 28) || (uint32_t)((uint64_t)den >> 32) - ((1u << 28) + 1u) >= (1u << 29) - 1u)
        return false;
    if (want) {
        mom[0] = dd;
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            double jd = diff_to_double((uint64_t)j[d], 0);
            if (REG && ((k.mask >> d) & 1u)) jd = fma(0.5 * a[d], dd, jd);
            mom[1 + d] = inv * jd;
            if (!REG && ((k.mask >> d) & 1u)) mom[1 + d] = fma(0.5, a[d], mom[1 + d]);
        }
    }
    // S (2^59): xx, yy, zz, xy, xz, yz
    const Fix2 ux = digits(u[0] + k.k[0]), uy = digits(u[1] + k.k[1]), uz = digits(u[2] + k.k[2]);
    int64_t sxx = mulq(sd[0], ux), syy = mulq(sd[1], uy), szz = mulq(sd[2], uz);
    int64_t sxy = mulq(sd[0], uy), sxz = mulq(sd[0], uz), syz = mulq(sd[1], uz);
    if (k.mask & 1u) {
        sxx += mulq(sd[0], k.k2[0]);
        sxy += mulq(sd[1], k.k2[0]);
        sxz += mulq(sd[2], k.k2[0]);
    }
    if (k.mask & 2u) {
        syy += mulq(sd[1], k.k2[1]);
        syz += mulq(sd[2], k.k2[1]);
    }
    if (k.mask & 4u) szz += mulq(sd[2], k.k2[2]);
    // a den / wo (regularized: a den) for the odd parts
    int64_t t[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        t[d] = j[d];
        if ((k.mask >> d) & 1u) t[d] += mulq(dn, k.ao[d]);
    }
    uint32_t low = 0;
    if (!REG) {
        const int64_t base = 3 * (sxx + syy + szz) - (den >> 1);
        int64_t sum = 0;
        auto pair = [&](int i, int64_t y, int64_t b, int64_t odd) {
            const int64_t E = mulq<0, DOWN>(9 * (fe[i] - y) + b, k.e);
            const int64_t O = mulq<0, DOWN>(6 * fo[i] - odd, k.o);
            sum += E;
            f[8 - i] = round_to_double(x[8 - i] - E + O, low);
            f[10 + i] = round_to_double(x[10 + i] - E - O, low);
        };
        pair(6, 2 * sxx, 2 * base, 2 * t[0]);
        pair(2, 2 * syy, 2 * base, 2 * t[1]);
        pair(0, 2 * szz, 2 * base, 2 * t[2]);
        const int64_t dxy = sxx + syy, dxz = sxx + szz, dyz = syy + szz;
        pair(8, dxy + 2 * sxy, base, t[0] + t[1]);
        pair(4, dxy - 2 * sxy, base, t[0] - t[1]);
        pair(7, dxz + 2 * sxz, base, t[0] + t[2]);
        pair(5, dxz - 2 * sxz, base, t[0] - t[2]);
        pair(3, dyz + 2 * syz, base, t[1] + t[2]);
        pair(1, dyz - 2 * syz, base, t[1] - t[2]);
        f[9] = round_to_double(x[9] + 2 * sum, low);
    } else {
        // 3 H2 (2^57) from 3 P and 3 S: any mix of populations in range stays
        // below 2^63, and a last place there is 2^-62 of a population
        auto relaxed = [&](int64_t p3, int64_t s59) {
            const int64_t p = (p3 + 8) >> 4, s = (3 * s59 + 2) >> 2;
            return p + mulq<3>(digits(s - p), k.w);
        };
        const int64_t xx = relaxed(3 * ((fe[4] + fe[5]) + (fe[6] + fe[7]) + fe[8]) - den, sxx);
        const int64_t yy = relaxed(3 * ((fe[1] + fe[2]) + (fe[3] + fe[4]) + fe[8]) - den, syy);
        const int64_t zz = relaxed(3 * ((fe[0] + fe[1]) + (fe[3] + fe[5]) + fe[7]) - den, szz);
        const int64_t xy = relaxed(3 * (fe[8] - fe[4]), sxy), xz = relaxed(3 * (fe[7] - fe[5]), sxz);
        const int64_t yz = relaxed(3 * (fe[3] - fe[1]), syz);
        const int64_t base = ((den + 4) >> 3) - (xx + yy + zz); // 2 den - 3 tr H2
        int64_t sum = 0;
        auto pair = [&](int i, int64_t v, int64_t odd) {
            const int64_t e = mulq<0, DOWN>(v, k.c72), o = mulq<0, DOWN>(odd, k.c12);
            sum += e;
            f[8 - i] = round_to_double(e - o, low);
            f[10 + i] = round_to_double(e + o, low);
        };
        pair(6, 2 * base + 6 * xx, 2 * t[0]);
        pair(2, 2 * base + 6 * yy, 2 * t[1]);
        pair(0, 2 * base + 6 * zz, 2 * t[2]);
        const int64_t dxy = base + 3 * (xx + yy), dxz = base + 3 * (xx + zz), dyz = base + 3 * (yy + zz);
        pair(8, dxy + 6 * xy, t[0] + t[1]);
        pair(4, dxy - 6 * xy, t[0] - t[1]);
        pair(7, dxz + 6 * xz, t[0] + t[2]);
        pair(5, dxz - 6 * xz, t[0] - t[2]);
        pair(3, dyz + 6 * yz, t[1] + t[2]);
        pair(1, dyz - 6 * yz, t[1] - t[2]);
        f[9] = round_to_double(den - 2 * sum, low);
    }
    return low < (1u << 31) - (1u << 20);
}

} // namespace jlb
