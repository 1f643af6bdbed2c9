// lbm_fp64.cu -- FP64 time step with the reference's arithmetic.
//
// This translation unit is compiled with -fmad=false: every FP64 operation
// below is a separately rounded IEEE add/mul/div written in the order the
// reference evaluates it (jyulb/D3Q19.pyx:348-940, jyulb/bcs.pyx:31-716,
// jyulb/isothermal.pyx:1112-1248), so the GPU reproduces the reference's
// populations and moments bit for bit on x86-64 builds of the reference.
#include "lbm_fp64.cuh"

namespace jlb {

// What bounds this step is the FP64 pipe: GB300 issues one FP64 warp
// instruction per 16-19 cycles and SM (an integer one takes half a cycle), so
// the collision is written for the fewest FP64 operations that still round
// like the reference's:
//   * products by powers of two are exact, so x +- 2 y is one FMA with a single
//     rounding, the reference's own; its 2 h, 6 h, 12 h and 18 h terms come
//     from 3 h and 6 h, and 4 h - 6 h sums share the halved sums of the others;
//   * constants of the rates and the uniform force come from the host
//     (StepArgs::k64, the same IEEE operations), not from every thread;
//   * terms of force components that are zero add zeros, and are left out;
//   * the bulk of the sites (collide_int) does the additions of the moments,
//     the reciprocal of the density, the products with constants and the sums
//     and differences of the projection's even and odd parts on the integer
//     pipes, beside the FP64 pipe: of about 210 FP64 operations of a TRT site
//     77 are left, and both kinds of pipe take about as long.
// Same bits as the plain form (collide_plain, which sites near overflow or
// underflow take).  128^3 cavity, us a step: plain; with integer
// moments and relaxation; with the reciprocal too; with the moments' and the
// projection's constants; with its sums; with the present range checks: TRT 1111,
// 562, 548, 490, 452, 440; BGK 938, 497, 479, 425, 383, 378; regularized 938, 521,
// 502, 402, 366, 366.
template <int SCH> struct Phys64 : Phys64Base {
    static constexpr bool host_consts = true;

    // one entry of the second-moment force c2 (a_p j_r + a_r j_p)
    __device__ static void force_off(C &h, C c2, unsigned p, unsigned r, C ap, C ar, C jp, C jr) {
        if (!(p | r)) return;
        C t;
        if (p && r) t = ap * jr + ar * jp;
        else t = p ? ap * jr : ar * jp;
        h = h + c2 * t;
    }
    // force terms of the moments (jyulb/D3Q19.pyx:655-940): first moments
    // with F.c1a = c1 a, second moments with c2; j is den u
    __device__ static void force(C *h, const Force64 &F, const Consts64 &k, C den, C jx, C jy, C jz) {
        const unsigned mx = F.mask & 1u, my = F.mask & 2u, mz = F.mask & 4u;
        if (mx) { h[1] = h[1] + F.c1a[0] * den; h[4] = h[4] + F.c2a[0] * jx; }
        if (my) { h[2] = h[2] + F.c1a[1] * den; h[7] = h[7] + F.c2a[1] * jy; }
        if (mz) { h[3] = h[3] + F.c1a[2] * den; h[9] = h[9] + F.c2a[2] * jz; }
        force_off(h[5], k.c2, mx, my, F.a[0], F.a[1], jx, jy);
        force_off(h[6], k.c2, mx, mz, F.a[0], F.a[2], jx, jz);
        force_off(h[8], k.c2, my, mz, F.a[1], F.a[2], jy, jz);
    }

    // Phys64Base::project with the reference's roundings and fewer operations
    template <bool ADD> __device__ static void project_fused(const C *h, C *f) {
        const C c = 1.0 / 72.0, cc = 2.0 * (1.0 / 72.0);
        const C t4 = 3.0 * h[4], t7 = 3.0 * h[7], t9 = 3.0 * h[9];
        const C s = h[0] + t4, v = __fma_rn(2.0, h[0], -t4);
        const C w = __fma_rn(2.0, s, -t7), v2 = __fma_rn(2.0, t7, v);
        const C exy = __fma_rn(2.0, s + t7, -t9), exz = __fma_rn(2.0, t9, w), eyz = __fma_rn(2.0, t9, v2);
        const C ex = w - t9, ey = v2 - t9, ez = __fma_rn(2.0, t9, v - t7); // halves of the reference's
        const C q1 = 6.0 * h[1], q2 = 6.0 * h[2], q3 = 6.0 * h[3];
        auto put = [&](int q, C p) { f[q] = ADD ? f[q] + p : p; };
        auto pair = [&](int lo, C e, C o) { // f_lo from e - o, its opposite from e + o
            put(lo, c * (e - o));
            put(18 - lo, c * (e + o));
        };
        C o;
        o = 18.0 * h[5]; pair(0, exy + o, q1 + q2); pair(4, exy - o, q1 - q2);
        o = 18.0 * h[6]; pair(1, exz + o, q1 + q3); pair(3, exz - o, q1 - q3);
        o = 18.0 * h[8]; pair(5, eyz + o, q2 + q3); pair(7, eyz - o, q2 - q3);
        put(2, cc * (ex - q1)); put(16, cc * (ex + q1));
        put(6, cc * (ey - q2)); put(12, cc * (ey + q2));
        put(8, cc * (ez - q3)); put(10, cc * (ez + q3));
        put(9, __fma_rn(-0.5, h[4] + h[7] + h[9], (1.0 / 3.0) * h[0]));
    }

    // products with the positive constants of the rates and the projection:
    // integer ones in the integer form
    template <bool INT> __device__ static C times(C x, C k, const soft64::MulC &m) {
        if constexpr (INT) return soft64::mulz(x, m);
        else return x * k;
    }
    // relaxed moments of BGK / TRT from den and the stored velocity
    template <bool INT> __device__ static void relaxed_moments(C *h, const Force64 &F, const Consts64 &k, C den, C &ux, C &uy, C &uz) {
        if (F.mask & 1u) ux = __fma_rn(0.5, F.a[0], ux);
        if (F.mask & 2u) uy = __fma_rn(0.5, F.a[1], uy);
        if (F.mask & 4u) uz = __fma_rn(0.5, F.a[2], uz);
        const C jx = den * ux, jy = den * uy, jz = den * uz;
        h[0] = times<INT>(den, k.we, k.mwe);
        h[1] = times<INT>(jx, k.wodd, k.mwo); h[2] = times<INT>(jy, k.wodd, k.mwo); h[3] = times<INT>(jz, k.wodd, k.mwo);
        h[4] = times<INT>(jx * ux, k.we, k.mwe); h[5] = times<INT>(jx * uy, k.we, k.mwe);
        h[6] = times<INT>(jx * uz, k.we, k.mwe); h[7] = times<INT>(jy * uy, k.we, k.mwe);
        h[8] = times<INT>(jy * uz, k.we, k.mwe); h[9] = times<INT>(jz * uz, k.we, k.mwe);
        force(h, F, k, den, jx, jy, jz);
    }
    // regularized: h holds the moments of f; relaxes them and sets the
    // stored velocity
    template <bool INT>
    __device__ static void relaxed_moments_reg(C *h, const Force64 &F, const Consts64 &k, C inv, C &ux, C &uy, C &uz) {
        const C den = h[0];
        C jx = h[1], jy = h[2], jz = h[3];
        if (F.mask & 1u) jx = __fma_rn(0.5, F.a[0] * den, jx);
        if (F.mask & 2u) jy = __fma_rn(0.5, F.a[1] * den, jy);
        if (F.mask & 4u) jz = __fma_rn(0.5, F.a[2] * den, jz);
        ux = inv * jx; uy = inv * jy; uz = inv * jz;
        const C ex = den * ux, ey = den * uy, ez = den * uz;
        const C he[10] = {den, ex, ey, ez, ex * ux, ex * uy, ex * uz, ey * uy, ey * uz, ez * uz};
#pragma unroll
        for (int m = 0; m < 10; ++m) {
            const C e = times<INT>(he[m], k.we, k.mwe);
            if (INT && !(k.nonzero & 4u)) h[m] = e; // 1 - we = 0
            else h[m] = times<INT>(h[m], k.r9, k.mr9) + e;
        }
        force(h, F, k, den, jx, jy, jz);
    }

    // The update in the reference's own operations (jyulb/D3Q19.pyx:655-940).
    // project_fused halves and doubles where the reference multiplies, and skips
    // terms of zero force, which is the same until a number overflows, becomes
    // denormal, or is not finite; ordinary() tells.
    __device__ __noinline__ static C collide_plain(C *f, const Force64 &F, const Consts64 &k, C *u) {
        const C ax = F.a[0], ay = F.a[1], az = F.a[2], we = k.we, wo = k.wodd;
        C h[10];
        if (SCH != SCH_REG) {
            const C c2 = 1.0 - 0.5 * we, c1 = SCH == SCH_TRT ? 1.0 - 0.5 * wo : c2;
            const C den = f_to_den_vel(f, u[0], u[1], u[2]);
            u[0] = u[0] + 0.5 * ax; u[1] = u[1] + 0.5 * ay; u[2] = u[2] + 0.5 * az;
            heq(den, u[0], u[1], u[2], h);
#pragma unroll
            for (int m = 0; m < 10; ++m) h[m] = h[m] * (m >= 1 && m <= 3 ? wo : we);
            const C jx = den * u[0], jy = den * u[1], jz = den * u[2];
            h[1] = h[1] + c1 * ax * den; h[2] = h[2] + c1 * ay * den; h[3] = h[3] + c1 * az * den;
            force_h2(h, c2, ax, ay, az, jx, jy, jz);
            relax(f, k);
            project<true>(h, f);
            return den;
        } else {
            const C c2 = 1.0 - 0.5 * we;
            C he[10];
            f_to_h(f, h);
            const C den = h[0], inv = 1.0 / den;
            const C jx = h[1] + 0.5 * ax * den, jy = h[2] + 0.5 * ay * den, jz = h[3] + 0.5 * az * den;
            u[0] = inv * jx; u[1] = inv * jy; u[2] = inv * jz;
            heq(den, u[0], u[1], u[2], he);
#pragma unroll
            for (int m = 0; m < 10; ++m) h[m] = h[m] * k.r9 + we * he[m];
            h[1] = h[1] + c2 * ax * den; h[2] = h[2] + c2 * ay * den; h[3] = h[3] + c2 * az * den;
            force_h2(h, c2, ax, ay, az, jx, jy, jz);
            project<false>(h, f);
            return den;
        }
    }
    // density in [2^-100, 2^100) and velocity components that are zero or in
    // [2^-200, 2^200) (regularized: momenta and second moments): with the bounds
    // of Force64::plain every product and sum of the update is then zero or in
    // [2^-900, 2^1000)
    template <int N> __device__ static bool ordinary(C den, const C *x) {
        const uint32_t e = (uint32_t)(soft64::bits(den) >> 52) & 0x7ffu;
        bool ok = e - (1023u - 100u) < 200u;
#pragma unroll
        for (int i = 0; i < N; ++i) ok = ok && zero_or_within(x[i], -200, 200);
        return ok;
    }
    __device__ static C plain_site(C *f, const Force64 &F, const Consts64 &k, C &ux, C &uy, C &uz) {
        C g[Q], u[3]; // collide_plain takes addresses
#pragma unroll
        for (int q = 0; q < Q; ++q) g[q] = f[q];
        const C den = collide_plain(g, F, k, u);
#pragma unroll
        for (int q = 0; q < Q; ++q) f[q] = g[q];
        ux = u[0]; uy = u[1]; uz = u[2];
        return den;
    }

    // f_q <- c3 f_q - c4 f_opp (BGK: (1 - we) f_q)
    __device__ static void relax(C *f, const Consts64 &k) {
        if (SCH == SCH_BGK) {
#pragma unroll
            for (int q = 0; q < Q; ++q) f[q] = f[q] * k.r9;
        } else {
#pragma unroll
            for (int q = 0; q < 9; ++q) {
                const C fa = f[q], fb = f[18 - q];
                f[q] = k.c3 * fa - k.c4 * fb;
                f[18 - q] = k.c3 * fb - k.c4 * fa;
            }
            f[9] = f[9] * k.r9;
        }
    }
    // moments of f (jyulb/D3Q19.pyx:395-452)
    __device__ static void f_to_h(const C *f, C *h) {
        C d1x = f[0] + f[1] + f[2] + f[3] + f[4];
        C dx1 = f[14] + f[15] + f[16] + f[17] + f[18];
        C d01y = f[5] + f[6] + f[7];
        C d0y1 = f[11] + f[12] + f[13];
        C d1y = f[0] + d01y + f[14];
        C dy1 = f[4] + d0y1 + f[18];
        C d1z = f[1] + f[5] + f[8] + f[11] + f[15];
        C dz1 = f[3] + f[7] + f[10] + f[13] + f[17];
        C den = d1x + dx1 + d01y + d0y1 + f[8] + f[9] + f[10];
        h[0] = den; h[1] = dx1 - d1x; h[2] = dy1 - d1y; h[3] = dz1 - d1z;
        const C d3 = (1.0 / 3.0) * den;
        h[4] = (d1x + dx1) - d3;
        h[5] = f[0] + f[18] - f[4] - f[14];
        h[6] = f[1] + f[17] - f[3] - f[15];
        h[7] = (d1y + dy1) - d3;
        h[8] = f[5] + f[13] - f[7] - f[11];
        h[9] = (d1z + dz1) - d3;
    }

    // forward-Euler update; returns den, writes the stored velocity
    // u = j/den + a/2 (jyulb/D3Q19.pyx:655-940)
    __device__ static C collide(C *f, const Force64 &F, const Consts64 &k, C &ux, C &uy, C &uz) {
        C h[10];
        if (SCH != SCH_REG) {
            const C den = f_to_den_vel(f, ux, uy, uz);
            const C u[3] = {ux, uy, uz};
            if (F.plain || !ordinary<3>(den, u)) return plain_site(f, F, k, ux, uy, uz);
            relaxed_moments<false>(h, F, k, den, ux, uy, uz);
            relax(f, k);
            project_fused<true>(h, f);
            return den;
        } else {
            f_to_h(f, h);
            if (F.plain || !ordinary<9>(h[0], h + 1)) return plain_site(f, F, k, ux, uy, uz);
            const C den = h[0];
            relaxed_moments_reg<false>(h, F, k, 1.0 / h[0], ux, uy, uz);
            project_fused<false>(h, f);
            return den;
        }
    }
    // the FP64 form of a site that collide_int refuses, out of line: inline, the
    // accepted sites lose (128^3, us a step: BGK 362 -> 375, TRT 433 -> 450)
    __device__ __noinline__ static C collide_cold(C *f, const Force64 &F, const Consts64 &k, C *u) {
        return collide(f, F, k, u[0], u[1], u[2]);
    }

    // What collide_int's range leaves the rest population, near equilibrium.
    // Looked at before anything else, so that a site with a density far from 1
    // pays for nothing but the FP64 form.
    __device__ static bool int_range(const C *f) { return soft64::within(f[9], 0x1p-5, 1.5); }

    // The same update, with most of its operations on the integer pipes
    // (soft64.cuh): the same bits.  It needs populations in [2^-9, 1/4) (rest:
    // int_range(); the sum then stays below 2^64 units), velocities that are zero
    // or in [2^-400, 2^8), and projections whose even parts outweigh the odd ones;
    // anything else sets `bad` and leaves f undefined.
    __device__ static C collide_int(C *f, const Force64 &F, const Consts64 &k, C &ux, C &uy, C &uz, bool &bad) {
        using namespace soft64;
        C h[10], den, inv;
        uint32_t range = 0, rest = 0, least = 0;
        {
            uint64_t x[Q];
#pragma unroll
            for (int q = 0; q < Q; ++q) x[q] = fix(f[q], q == 9 ? rest : range);
            const uint64_t d1x = add(add(add(add(x[0], x[1]), x[2]), x[3]), x[4]);
            const uint64_t dx1 = add(add(add(add(x[14], x[15]), x[16]), x[17]), x[18]);
            const uint64_t d01y = add(add(x[5], x[6]), x[7]);
            const uint64_t d0y1 = add(add(x[11], x[12]), x[13]);
            const uint64_t xx = add(d1x, dx1);
            const uint64_t xd = add(add(add(add(add(xx, d01y), d0y1), x[8]), x[9]), x[10]);
            den = to_double(xd);
            inv = recip(xd);
            const C jx = diff_to_double(dx1, d1x);
            if (SCH != SCH_REG) {
                // jyulb/D3Q19.pyx:348-390
                const uint64_t y = sub(sub(add(add(x[4], d0y1), x[18]), x[0], least), d01y, least);
                const uint64_t zp = add(add(add(add(x[3], x[7]), x[10]), x[13]), x[17]);
                const uint64_t z = sub(sub(sub(sub(zp, x[1], least), x[5], least), x[8], least), x[11], least);
                const C jy = diff_to_double(y, x[14]), jz = diff_to_double(z, x[15]);
                ux = inv * jx; uy = inv * jy; uz = inv * jz;
            } else {
                // jyulb/D3Q19.pyx:395-452
                const uint64_t d1y = add(add(x[0], d01y), x[14]), dy1 = add(add(x[4], d0y1), x[18]);
                const uint64_t d1z = add(add(add(add(x[1], x[5]), x[8]), x[11]), x[15]);
                const uint64_t dz1 = add(add(add(add(x[3], x[7]), x[10]), x[13]), x[17]);
                const C d3 = (1.0 / 3.0) * den;
                h[0] = den; h[1] = jx; h[2] = diff_to_double(dy1, d1y); h[3] = diff_to_double(dz1, d1z);
                h[4] = to_double(xx) - d3;
                h[5] = diff_to_double(sub(add(x[0], x[18]), x[4], least), x[14]);
                h[6] = diff_to_double(sub(add(x[1], x[17]), x[3], least), x[15]);
                h[7] = to_double(add(d1y, dy1)) - d3;
                h[8] = diff_to_double(sub(add(x[5], x[13]), x[7], least), x[11]);
                h[9] = to_double(add(d1z, dz1)) - d3;
            }
        }
        if (SCH != SCH_REG) {
            relaxed_moments<true>(h, F, k, den, ux, uy, uz);
            if (SCH == SCH_BGK) {
                // 1 - we = 0 (tau = 1) leaves the projection alone
                if (k.nonzero & 4u) {
#pragma unroll
                    for (int q = 0; q < Q; ++q) f[q] = mul(f[q], k.mr9);
                } else {
#pragma unroll
                    for (int q = 0; q < Q; ++q) f[q] = 0.0;
                }
            } else {
                if (!(k.nonzero & 3u)) { // c3 = c4 = 0 (both rates 1)
#pragma unroll
                    for (int q = 0; q < Q; ++q) if (q != 9) f[q] = 0.0;
                } else if (!(k.nonzero & 1u)) { // c3 = 0: 0 - c4 f
#pragma unroll
                    for (int q = 0; q < 9; ++q) {
                        const C fa = f[q], fb = f[18 - q];
                        f[q] = -mul(fb, k.mc4);
                        f[18 - q] = -mul(fa, k.mc4);
                    }
                } else if (!(k.nonzero & 2u)) { // c4 = 0 (equal rates)
#pragma unroll
                    for (int q = 0; q < 9; ++q) {
                        f[q] = mul(f[q], k.mc3);
                        f[18 - q] = mul(f[18 - q], k.mc3);
                    }
                } else {
#pragma unroll
                    for (int q = 0; q < 9; ++q) {
                        const C fa = f[q], fb = f[18 - q];
                        f[q] = mul(fa, k.mc3) - mul(fb, k.mc4);
                        f[18 - q] = mul(fb, k.mc3) - mul(fa, k.mc4);
                    }
                }
                f[9] = k.nonzero & 4u ? mul(f[9], k.mr9) : 0.0;
            }
        } else {
            relaxed_moments_reg<true>(h, F, k, inv, ux, uy, uz);
        }
        uint32_t span = 0;
        int32_t apart = 1 << 30, close = 1 << 30;
        project_int<SCH != SCH_REG>(h, k, f, span, apart, close);
        // velocities are zero or in [2^-400, 2^8): their products, and those
        // with the force they bound, are normal.  An acceleration field may hold
        // anything; mul() of a NaN or an infinity would be some finite number
        uint32_t beyond = 0;
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            const uint64_t u = bits(d == 0 ? ux : d == 1 ? uy : uz);
            const uint32_t e = (uint32_t)(u >> 52) & 0x7ffu;
            const uint32_t z = (u << 1) ? e - (1023u - 400u) : 0u;
            beyond = beyond > z ? beyond : z;
        }
        bad = range > 6u || least >= (1u << 31) - (1u << 21) || span > PROJ_SPAN || apart < 0 || close < 1 << 21 ||
              beyond > 407u;
        return den;
    }

    // project_fused with integer products and sums; `span` exceeds PROJ_SPAN
    // unless every even part lies in [2^-40, 2^10); `apart` is negative or `close`
    // below 2^21 where an odd part is not smaller than its even one, or reaches it
    // but for 2^-8 of the even one's binade
    static constexpr uint32_t PROJ_LO = (1023u - 40u) << 20, PROJ_SPAN = (50u << 20) - 1u;
    template <bool ADD>
    __device__ static void project_int(const C *h, const Consts64 &k, C *f, uint32_t &span, int32_t &apart, int32_t &close) {
        const C t4 = soft64::mulz(h[4], k.m3), t7 = soft64::mulz(h[7], k.m3), t9 = soft64::mulz(h[9], k.m3);
        const C s = h[0] + t4, v = __fma_rn(2.0, h[0], -t4);
        const C w = __fma_rn(2.0, s, -t7), v2 = __fma_rn(2.0, t7, v);
        const C exy = __fma_rn(2.0, s + t7, -t9), exz = __fma_rn(2.0, t9, w), eyz = __fma_rn(2.0, t9, v2);
        const C ex = w - t9, ey = v2 - t9, ez = __fma_rn(2.0, t9, v - t7);
        const C q1 = soft64::mulz(h[1], k.m6), q2 = soft64::mulz(h[2], k.m6), q3 = soft64::mulz(h[3], k.m6);
        auto put = [&](int q, C p) { f[q] = ADD ? f[q] + p : p; };
        auto both = [&](int lo, C e, C o, const soft64::MulC &m) { // f_lo from e - o, its opposite from e + o
            const uint32_t x = (uint32_t)__double2hiint(e) - PROJ_LO;
            span = span > x ? span : x;
            C plus, minus;
            soft64::add_sub(e, o, plus, minus, apart, &close);
            put(lo, soft64::mul(minus, m));
            put(18 - lo, soft64::mul(plus, m));
        };
        C o;
        o = soft64::mulz(h[5], k.m18); both(0, exy + o, q1 + q2, k.m72); both(4, exy - o, q1 - q2, k.m72);
        o = soft64::mulz(h[6], k.m18); both(1, exz + o, q1 + q3, k.m72); both(3, exz - o, q1 - q3, k.m72);
        o = soft64::mulz(h[8], k.m18); both(5, eyz + o, q2 + q3, k.m72); both(7, eyz - o, q2 - q3, k.m72);
        both(2, ex, q1, k.m36); both(6, ey, q2, k.m36); both(8, ez, q3, k.m36);
        put(9, __fma_rn(-0.5, h[4] + h[7] + h[9], (1.0 / 3.0) * h[0]));
    }
};

int launch_step_fp64(const StepArgs &a, int scheme, bool pstep, bool accf, int blocks, cudaStream_t st) {
    return launch_step_impl<StoreF64, Phys64>(a, scheme, pstep, accf, blocks, st);
}

} // namespace jlb
