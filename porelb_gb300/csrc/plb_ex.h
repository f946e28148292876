/*
 * plb_ex.h - the bit-exact BGK collision, most of its IEEE operations done
 * on the integer pipes.
 *
 * The bit-exact form rounds every operation of porelb.c:318-365 as FP64
 * hardware does.  GB300 issues an FP64 operation of a warp about every 20
 * clocks of an SM, an integer one every half clock, so even a dozen integer
 * instructions per rounded operation are the cheaper way.  What makes them
 * a dozen and not fifty is that the collision's values are near the lattice
 * weights: they are held as fixed-point integers whose binade is known to
 * within a few places, so an IEEE add is an integer add and a rounding to
 * nearest even at a bit that one shift or one leading-zero count gives, and
 * a product one 2x2-limb multiply and the same rounding.  No operand is
 * unpacked from or packed to its FP64 bits between two operations.
 *
 *   f_j        class scale: f * 2^(62 + s), s = 1, 4, 5 for the weights 1/3,
 *              1/18, 1/36 (weights near 2^62), and Q61 for the sums
 *   rho        Q61, rounded at each of the reference's 18 adds
 *   j = sum e f  Q61; every partial sum is exact (and so is IEEE's) when it
 *              stays below 2^-5 and the f are multiples of 2^-58; else the
 *              27 adds run natively
 *   u          integer quotients, corrected by their exact remainders
 *   1 + 3 e.u + 4.5 (e.u)^2 - 1.5 u.u   Q62, rounded after each add
 *   feq, (omega + a) feq, (1 - omega) f, their sum   class scale
 *
 * A value that is shifted below the last place kept leaves a sticky one in
 * it (rounding to odd), which preserves any later rounding to nearest at a
 * place at least two bits higher (Boldo & Melquiond 2008).  The operations
 * whose operands can have any exponent (u.u, e.u, 4.5 (e.u)^2, the forcing
 * factor) stay on the FP64 pipe, and so does the last rounding, as its
 * integer-to-FP64 conversion: about 65 of a node's 260.
 *
 * Domain (anything else is reported and the caller takes another path):
 * f_0 in [1/4, 1), f_1..6 in [2^-7, 2^-3), f_7..18 in [2^-8, 2^-4), rho in
 * [1/2, 1.2], |u_a| < 0.11, omega + a in [1/8, 2) for every direction (or,
 * for a large tau, in a range 16 times as wide from its lower end to its upper
 * that is a power of two lower), and 1 - omega zero or of magnitude >= 2^-40.
 * A node that is outside by its velocity alone is told apart: its moments
 * stand.
 *
 * Measured (256^3 pack, 5.87M nodes): 990 us a step (5.9 GLUPS) against 2204
 * (2.66) with every add on the FP64 pipe and IEEE products made one by one
 * from FP64 bits; 24x20x16: 8.7 against 15 us.  Bound by the integer ALU and
 * FP64 pipes together, each about three quarters busy.
 *
 * Host+device: a CPU build checks it bit for bit against FP64 arithmetic.
 */
#ifndef PLB_EX_H_
#define PLB_EX_H_

#include <math.h>
#include <stdint.h>
#include <string.h>

#if defined(__CUDACC__)
#define EX_HD __host__ __device__ __forceinline__
#else
#define EX_HD static inline
#endif

namespace plb {
namespace ex_ {

EX_HD uint64_t bits_of(double x)
{
#if defined(__CUDA_ARCH__)
    return (uint64_t)__double_as_longlong(x);
#else
    uint64_t u;
    memcpy(&u, &x, 8);
    return u;
#endif
}
EX_HD double of_bits(uint64_t u)
{
#if defined(__CUDA_ARCH__)
    return __longlong_as_double((long long)u);
#else
    double x;
    memcpy(&x, &u, 8);
    return x;
#endif
}
/* single rounded operations (the host build is compiled without contraction) */
#if defined(__CUDA_ARCH__)
EX_HD double add(double a, double b) { return __dadd_rn(a, b); }
EX_HD double sub(double a, double b) { return __dsub_rn(a, b); }
EX_HD double mul(double a, double b) { return __dmul_rn(a, b); }
#else
EX_HD double add(double a, double b) { return a + b; }
EX_HD double sub(double a, double b) { return a - b; }
EX_HD double mul(double a, double b) { return a * b; }
#endif

EX_HD uint32_t hi32(uint64_t x) { return (uint32_t)(x >> 32); }

/* leading zeros of x != 0 */
EX_HD uint32_t clz32(uint32_t x)
{
#if defined(__CUDA_ARCH__)
    return (uint32_t)__clz((int)x);
#else
    return (uint32_t)__builtin_clz(x);
#endif
}

EX_HD uint64_t mulhi64(uint64_t a, uint64_t b)
{
#if defined(__CUDA_ARCH__)
    return __umul64hi(a, b);
#else
    return (uint64_t)(((unsigned __int128)a * b) >> 64);
#endif
}

EX_HD uint32_t umax(uint32_t a, uint32_t b) { return a > b ? a : b; }
EX_HD uint32_t umin(uint32_t a, uint32_t b) { return a < b ? a : b; }
EX_HD int32_t imax(int32_t a, int32_t b) { return a > b ? a : b; }
EX_HD int32_t imin(int32_t a, int32_t b) { return a < b ? a : b; }

/* v rounded to nearest, ties to even, at bit d (1 <= d < 32): a multiple of
 * 2^d */
EX_HD uint64_t rne(uint64_t v, uint32_t d)
{
    const uint32_t M = (1u << d) - 1u;
    const uint64_t r = v + ((M >> 1) + (((uint32_t)v >> d) & 1u));
    return r & ~(uint64_t)M;
}

/* a * b / 2^64 rounded to nearest even at 53 significant bits, in place, for
 * a product in [2^117, 2^127) and (a >> 32) + (b >> 32) < 2^32 (which keeps
 * the sum of the middle products below 2^64).  The 64 bits below enter as
 * one: with the kept part's last bit they decide a tie. */
EX_HD uint64_t mulr(uint64_t a, uint64_t b)
{
    const uint32_t al = (uint32_t)a, ah = hi32(a), bl = (uint32_t)b, bh = hi32(b);
    const uint64_t ll = (uint64_t)al * bl;
    uint64_t mid = (uint64_t)ah * bl + hi32(ll);
    mid += (uint64_t)al * bh;
    const uint64_t top = (uint64_t)ah * bh + hi32(mid);
    const uint32_t below = umin((uint32_t)mid | (uint32_t)ll, 1u);
    const uint32_t c = clz32(hi32(top)); /* the last place is bit 11 - c */
    const uint32_t r = ((uint32_t)top >> ((11u - c) & 31u) | below) & 1u;
    return (top + ((0x3ffu >> c) + r)) & ~(uint64_t)(0x7ffu >> c);
}

/* the significand (with its leading one) of a normal FP64 value, as bits */
EX_HD uint64_t mant(uint64_t b)
{
    return (b & 0xfffffffffffffull) | 0x10000000000000ull;
}
EX_HD uint32_t expo(uint64_t b) { return hi32(b) >> 20; } /* of a positive value */

/* v >> s and (v >> s) << s; zero for s > 63 */
EX_HD uint64_t shr(uint64_t v, uint32_t s)
{
#if defined(__CUDA_ARCH__)
    uint64_t r;
    asm("shr.u64 %0, %1, %2;" : "=l"(r) : "l"(v), "r"(s));
    return r;
#else
    return s > 63u ? 0ull : v >> s;
#endif
}
EX_HD uint64_t shl(uint64_t v, uint32_t s)
{
#if defined(__CUDA_ARCH__)
    uint64_t r;
    asm("shl.b64 %0, %1, %2;" : "=l"(r) : "l"(v), "r"(s));
    return r;
#else
    return s > 63u ? 0ull : v << s;
#endif
}

/* v / 2^s rounded to odd */
EX_HD uint64_t shr_odd(uint64_t v, uint32_t s)
{
    const uint64_t q = shr(v, s);
    return q | (uint64_t)(shl(q, s) != v);
}

/* x in Q62 rounded to odd, for 0 <= x < 1/2 (a zero gives a sticky one,
 * which rounds away) */
EX_HD uint64_t q62(double x)
{
    const uint64_t b = bits_of(x);
    return shr_odd(mant(b) << 8, 1021u - (hi32(b) >> 20));
}

/* the FP64 product 3 x in Q62 rounded to odd, for 0 <= x < 1/4: three times
 * the significand, rounded to 53 bits */
EX_HD uint64_t q62_triple(double x)
{
    const uint64_t b = bits_of(x);
    const uint64_t m = 3ull * mant(b);
    const uint32_t g = hi32(m) >> 22; /* 1 if m >= 2^54 */
    const uint64_t r = (m + (g + (((uint32_t)m >> (1u + g)) & 1u))) & ~(uint64_t)(1u + 2u * g);
    return shr_odd(r << 8, 1021u - (hi32(b) >> 20));
}

/* x * 2^(62 + s) for class C's s, from the FP64 bits: no bit is lost for
 * the exponents of the domain */
EX_HD constexpr uint32_t kS(int c) { return c == 0 ? 1u : (c == 1 ? 4u : 5u); }
template <int C>
EX_HD uint64_t scaled(uint64_t b)
{
    return mant(b) << (expo(b) - (1013u - kS(C)) & 63u);
}

/* Per-run constants (host-computed). */
struct Consts {
    double omega, om1, k3, force, half_force;
    uint64_t om;   /* |1 - omega|'s significand, in [2^62, 2^63); 0 if omega = 1 */
    uint32_t omsh; /* |1 - omega| = om * 2^(-61 - ash - omsh) */
    uint32_t ash;  /* the forcing factor and the results are scaled 2^ash higher */
    uint32_t up;   /* the forcing factor is scaled 2^up higher still (TINY) */
    uint32_t neg;  /* 1 if 1 - omega < 0 */
    uint32_t ok;   /* the run's constants lie in the domain: 1, or 2 for TINY */
};

static inline Consts make_consts(double omega, double om1, double k3, double force,
                                 double half_force)
{
    Consts k;
    memset(&k, 0, sizeof(k));
    k.omega = omega;
    k.om1 = om1;
    k.k3 = k3;
    k.force = force;
    k.half_force = half_force;
    uint64_t b;
    memcpy(&b, &om1, 8);
    const uint32_t e = (uint32_t)(b >> 52) & 0x7ffu;
    k.ok = om1 == 0.0 || (e <= 1022u && e >= 983u);
    if (om1 != 0.0) k.om = mant(b) << 10;
    k.omsh = om1 != 0.0 ? 1024u - e : 0u;
    if (k.ok && k.omsh > 5u) k.ok = 2u;
    /* the forcing factor's bounds for any node (each node checks its own);
     * tau > 2.5 has 1 - omega in [0.6, 1): two places up fit */
    const double far = 1.11 * fabs(k3 * force);
    if (omega + far < 0.4) {
        k.ash = 2u;
        k.omsh -= 2u;
    }
    if (k.ok && k.ash && !(omega - far >= 0.03125)) {
        /* tau > 32: the factor with its own scale, its product shifted back.
         * (1 - omega) f is whole at the two places that are left, so the
         * sticky one of the sum is the product's alone */
        k.ok = 2u;
        k.omsh += k.ash;
        k.ash = 0u;
        while (k.up < 40u && omega + far < ldexp(1.0, -(int)k.up)) k.up++;
        if (!(omega - far >= ldexp(0.125, -(int)k.up) && omega + far < ldexp(2.0, -(int)k.up)))
            k.ok = 0u;
    } else if (!(omega - far >= (k.ash ? 0.03125 : 0.125) && omega + far < 2.0)) {
        k.ok = 0u;
    }
    k.neg = om1 < 0.0;
    return k;
}

EX_HD constexpr int xx(int j)
{
    return (j == 1 || j == 12 || j == 14 || j == 16 || j == 18) ? 1
         : (j == 2 || j == 11 || j == 13 || j == 15 || j == 17) ? -1 : 0;
}
EX_HD constexpr int xy(int j)
{
    return (j == 3 || j == 7 || j == 10 || j == 15 || j == 18) ? 1
         : (j == 4 || j == 8 || j == 9 || j == 16 || j == 17) ? -1 : 0;
}
EX_HD constexpr int xz(int j)
{
    return (j == 5 || j == 7 || j == 9 || j == 12 || j == 13) ? 1
         : (j == 6 || j == 8 || j == 10 || j == 11 || j == 14) ? -1 : 0;
}
EX_HD constexpr int xc(int j) { return j == 0 ? 0 : (j <= 6 ? 1 : 2); }
EX_HD double wt(int c) { return c == 0 ? 1.0 / 3 : (c == 1 ? 1.0 / 18 : 1.0 / 36); }

/* 2^126 / B to within a few units, for B in [2^63, 2^64): an FP32 reciprocal
 * and two Newton steps */
EX_HD uint64_t recip(uint64_t B)
{
    const uint32_t bh = hi32(B);
#if defined(__CUDA_ARCH__)
    const float r = __frcp_rn(__uint2float_rn(bh));
    const uint32_t rb = __float_as_uint(r);
#else
    const float r = 1.0f / (float)bh;
    uint32_t rb;
    memcpy(&rb, &r, 4);
#endif
    /* r in [2^-32, 2^-31]; x = r * 2^62 */
    const uint32_t x = ((rb & 0x7fffffu) | 0x800000u) << ((rb >> 23) - (127u - 32u) + 7u);
    /* 1 - B x / 2^94, in units of 2^-62 */
    const int64_t d0 = ((int64_t)1 << 62) -
                       (int64_t)((uint64_t)bh * x + (((uint64_t)(uint32_t)B * x) >> 32));
    const uint64_t I1 = ((uint64_t)x << 32) + (uint64_t)(((int64_t)(int32_t)(d0 >> 9) * (int64_t)x) >> 21);
    const int32_t d1 = (int32_t)(((int64_t)1 << 62) - (int64_t)mulhi64(B, I1));
    return I1 + (uint64_t)(((int64_t)d1 * (int64_t)hi32(I1)) >> 30);
}

/* x / rho, rounded to nearest: rho = b * 2^(eb - 1075) with b in [2^52,
 * 2^53), I = recip(b << 11).  The quotient of two 53-bit significands is
 * never halfway between two others, so the remainder of the rounded
 * estimate (exact modulo 2^64) says which neighbour is nearest. */
EX_HD double quotient(double x, uint64_t b, uint32_t eb, uint64_t I)
{
    const uint64_t xb = bits_of(x);
    const uint64_t m = mant(xb);
    const uint64_t q = mulhi64(m << 10, I); /* (m / b) * 2^61, within 4 */
    const uint32_t d = 8u + (hi32(q) >> 29);
    uint64_t r = (q + (64u << (d - 7u))) >> d;
    const int64_t rem = (int64_t)((m << (61u - d)) - r * b);
    r += (uint64_t)(2 * rem > (int64_t)b);
    r -= (uint64_t)(2 * rem < -(int64_t)b);
    const uint64_t y = ((uint64_t)(1013u + d + (expo(xb) & 0x7ffu) - eb) << 52) + r;
    return (xb << 1) == 0ull ? 0.0 : of_bits(y | (xb & 0x8000000000000000ull));
}

struct Out {
    double rho, u, v, w;
    uint32_t bad; /* density guard */
};

/* One collision.  b[19]: post-stream FP64 bits; store(j, bits) receives each
 * post-collision value as it is made (holding them to the end would cost the
 * registers of a third of the warps).  Returns kOutside or kFast when the node
 * lies outside the domain; store may then have received some values.  kFast:
 * o holds the moments all the same.  TINY: |1 - omega| < 1/16, whose products
 * can lose bits in the class scale and leave a sticky one, or k.up > 0, whose
 * products with the forcing factor can. */
constexpr uint32_t kOutside = 1u, kFast = 2u;

template <bool TINY, typename Store>
EX_HD uint32_t collide(const uint64_t (&b)[19], const Consts &k, bool it_pos, Out &o,
                       const Store &store)
{
    constexpr int Q = 19;
    /* range of the inputs */
    uint32_t lo1 = ~0u, hi1 = 0, lo2 = ~0u, hi2 = 0;
#pragma unroll
    for (int j = 1; j < Q; j++) {
        const uint32_t h = hi32(b[j]);
        if (xc(j) == 1) { lo1 = umin(lo1, h); hi1 = umax(hi1, h); }
        else { lo2 = umin(lo2, h); hi2 = umax(hi2, h); }
    }
    uint32_t outside = (uint32_t)(hi32(b[0]) - 0x3fd00000u >= 0x200000u) |
                       (uint32_t)(lo1 < 0x3f800000u) | (uint32_t)(hi1 >= 0x3fc00000u) |
                       (uint32_t)(lo2 < 0x3f700000u) | (uint32_t)(hi2 >= 0x3fb00000u);
    uint64_t F[Q]; /* class scale */
    F[0] = scaled<0>(b[0]);
#pragma unroll
    for (int j = 1; j < Q; j++) F[j] = xc(j) == 1 ? scaled<1>(b[j]) : scaled<2>(b[j]);

    /* rho in Q61, rounded at every add: its last place is bit 7, 8 or 9 */
    uint64_t S = F[0] >> 2;
    uint32_t low = 0;
    int64_t J[3] = {0, 0, 0};
    int32_t jmin = 0, jmax = 0;
#pragma unroll
    for (int j = 1; j < Q; j++) {
        const uint64_t f61 = F[j] >> (kS(xc(j)) + 1u);
        low |= (uint32_t)f61;
        S = rne(S + f61, 7u + (hi32(S + f61) >> 28));
        /* the momentum's partial sums */
#pragma unroll
        for (int a = 0; a < 3; a++) {
            const int e = a == 0 ? xx(j) : (a == 1 ? xy(j) : xz(j));
            if (e == 0) continue;
            J[a] = e > 0 ? J[a] + (int64_t)f61 : J[a] - (int64_t)f61;
            if (j <= 6 && (j & 1)) continue; /* the first term alone is an input */
            jmin = imin(jmin, (int32_t)hi32((uint64_t)J[a]));
            jmax = imax(jmax, (int32_t)hi32((uint64_t)J[a]));
        }
    }
    /* [1/2, 1.2], which is the density guard's range */
    outside |= (uint32_t)(S - ((uint64_t)1 << 60) > 0x1666666666666600ull);
    if (outside) return kOutside;
    o.bad = 0u;

    /* momentum: exact when every partial sum is below 2^-5 and a multiple of
     * 2^-58, else native adds */
    double m[3];
    if (jmin >= -(1 << 24) && jmax < (1 << 24) && (low & 7u) == 0u) {
#pragma unroll
        for (int a = 0; a < 3; a++) {
            const uint64_t c = bits_of((double)J[a]);
            m[a] = of_bits(J[a] == 0 ? 0ull : c - ((uint64_t)61 << 52));
        }
    } else {
#pragma unroll
        for (int a = 0; a < 3; a++) {
            double acc = 0.0;
            bool first = true;
#pragma unroll
            for (int j = 1; j < Q; j++) {
                const int e = a == 0 ? xx(j) : (a == 1 ? xy(j) : xz(j));
                if (e == 0) continue;
                /* the input back from its class scale (exact): keeping its
                 * bits alive to here would cost 36 registers */
                const double f =
                    of_bits(bits_of((double)(int64_t)F[j]) - ((uint64_t)(62u + kS(xc(j))) << 52));
                if (first) acc = e > 0 ? f : -f;
                else acc = e > 0 ? add(acc, f) : sub(acc, f);
                first = false;
            }
            m[a] = acc;
        }
    }
    if (it_pos) m[0] = add(m[0], k.half_force);

    /* rho's significand and exponent; u = j / rho */
    const uint32_t rd = 7u + (hi32(S) >> 28);
    const uint64_t rm = S >> rd;
    const uint32_t re = 1014u + rd;
    const uint64_t I = recip(rm << 11);
    const double u = quotient(m[0], rm, re, I), v = quotient(m[1], rm, re, I),
                 w = quotient(m[2], rm, re, I);
    const double rho = of_bits(((uint64_t)(re - 1u) << 52) + rm);
    o.rho = rho;
    o.u = u;
    o.v = v;
    o.w = w;
    {
        /* |u| < 0.11; j_x (the force's share can be any number) zero or far
         * from underflow */
        const uint32_t hu = hi32(bits_of(u)) & 0x7fffffffu, hv = hi32(bits_of(v)) & 0x7fffffffu,
                       hw = hi32(bits_of(w)) & 0x7fffffffu;
        const uint64_t jx = bits_of(m[0]) << 1;
        if (jx != 0ull && hi32(jx) < (128u << 20)) return kOutside;
        if (umax(umax(hu, hv), hw) >= 0x3fbc28f5u) return kFast;
    }

    const double uv = add(add(mul(u, u), mul(v, v)), mul(w, w));
    const uint64_t uv15 = q62(mul(1.5, uv));
    uint64_t h[3], A[3];
    {
        const double h0 = mul(wt(0), rho), h1 = mul(wt(1), rho), h2 = mul(wt(2), rho);
        h[0] = scaled<0>(bits_of(h0)) << 1;
        h[1] = scaled<1>(bits_of(h1)) << 1;
        h[2] = scaled<2>(bits_of(h2)) << 1;
        /* omega + ((1 - omega/2) 3 (e_x - u)) F for e_x = -1, 0, 1, Q62 */
#pragma unroll
        for (int e = -1; e <= 1; e++) {
            /* e = 0: the sign of a zero makes no difference to the sum */
            const double d = e == 0 ? -u : sub((double)e, u);
            const double a = add(k.omega, mul(mul(k.k3, d), k.force));
            const uint64_t ab = bits_of(a);
            const uint32_t s = TINY ? k.ash + k.up : k.ash;
            outside |= (uint32_t)(hi32(ab) - ((1020u - s) << 20) >= (4u << 20));
            A[e + 1] = mant(ab) << (expo(ab) + s - 1013u & 63u);
        }
    }
    if (outside) return kFast;

    uint32_t rmin = ~0u, rmax = 0;
    const uint64_t flip = (uint64_t)0 - k.neg;
    /* f' = (1 - omega) f + A feq from the equilibrium factor T (Q62) */
    auto relax = [&](int j, uint64_t T, uint64_t hc, uint64_t a) {
        /* feq * 2^(61 + s), the rest * 2^(59 + s + ash) */
        uint64_t R = mulr(a, mulr(hc, T));
        if (TINY) R = shr_odd(R, k.up);
        if (k.om != 0ull) {
            uint64_t p = mulr(k.om, F[j]);
            p = TINY ? shr_odd(p, k.omsh) : shr(p, k.omsh);
            R += (p ^ flip) + k.neg;
        }
        rmin = umin(rmin, hi32(R));
        if (TINY) rmax = umax(rmax, hi32(R));
        const uint32_t s = kS(xc(j));
        store(j, bits_of((double)(int64_t)R) - ((uint64_t)(59u + s + k.ash) << 52));
    };

    constexpr uint64_t kOne = (uint64_t)1 << 62;
    relax(0, kOne - rne(uv15, 9u), h[0], A[1]);
#pragma unroll
    for (int j = 1; j < Q; j += 2) {
        /* e.u of direction j as the reference adds it, its sign and
         * magnitude: the direction along it (plus) and the one against
         * (minus) */
        double eu = 0.0;
        bool first = true;
        if (xx(j) != 0) { eu = xx(j) > 0 ? u : -u; first = false; }
        if (xy(j) != 0) {
            const double t = xy(j) > 0 ? v : -v;
            eu = first ? t : add(eu, t);
            first = false;
        }
        if (xz(j) != 0) {
            const double t = xz(j) > 0 ? w : -w;
            eu = first ? t : add(eu, t);
            first = false;
        }
        const bool against = (hi32(bits_of(eu)) >> 31) != 0u; /* direction j is the minus one */
        eu = of_bits(bits_of(eu) & 0x7fffffffffffffffull);
        const uint64_t t3 = q62_triple(eu);
        const uint64_t c2 = q62(mul(mul(4.5, eu), eu));
        /* plus: 1 + t3 and + c2 are in [1, 2) (last place 2^-52); minus: 1 - t3
         * is exact where t3 >= 1/2, and then + c2 and - 1.5 u.u stay in
         * [1/2, 1] (2^-53), since 4.5 eu^2 < 3 |eu| and 1 - 6 a + 15 a^2 -
         * 1.5 a^2 > 1/2 for a < 0.111; - 1.5 u.u can bring the plus one below
         * 1 */
        const uint64_t p = kOne + rne(rne(t3, 10u) + c2, 10u) - uv15;
        const uint64_t n = kOne - rne(t3, 9u) + c2;
        const uint64_t Tp = rne(p, 9u + (hi32(p) >> 30));
        const uint64_t Tn = rne(rne(n, 9u) - uv15, 9u);
        relax(j, against ? Tn : Tp, h[xc(j)], A[xx(j) + 1]);
        relax(j + 1, against ? Tp : Tn, h[xc(j)], A[1 - xx(j)]);
    }
    /* exact integers convert whatever their size and sign, but zero; with a
     * sticky one they have to keep two bits below the last place */
    static_assert(kOutside == 1u, "");
    return TINY ? (uint32_t)(rmin < (1u << 24)) | (uint32_t)(rmax >= (1u << 28))
                : (uint32_t)(rmin == 0u);
}

}  // namespace ex_
}  // namespace plb

#endif
