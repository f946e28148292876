/* The integer bit-exact collision (plb_ex.h) against the same operations in
 * the host's FP64, one rounding each, bit for bit. */
#include <math.h>
#include <stdint.h>

#include "../../porelb_gb300/csrc/plb_ex.h"

using namespace plb;

namespace {

struct Rng {
    uint64_t s;
    uint64_t next()
    {
        uint64_t z = (s += 0x9E3779B97F4A7C15ull);
        z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
        z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
        return z ^ (z >> 31);
    }
    double u() { return (double)(next() >> 11) * 0x1p-53; }
    double sym() { return 2.0 * u() - 1.0; }
    bool one_in(int n) { return next() % (uint64_t)n == 0; }
};

const int *axis(int a)
{
    static int e[3][19];
    for (int j = 0; j < 19; j++) {
        e[0][j] = ex_::xx(j);
        e[1][j] = ex_::xy(j);
        e[2][j] = ex_::xz(j);
    }
    return e[a];
}

struct Macro {
    double rho, u[3];
    bool bad;
};

/* the collision of porelb.c:318-365 in its order of operations */
Macro reference(double (&f)[19], const ex_::Consts &k, bool it_pos)
{
    Macro m;
    m.rho = f[0];
    for (int j = 1; j < 19; j++) m.rho = m.rho + f[j];
    for (int a = 0; a < 3; a++) {
        const int *e = axis(a);
        double acc = 0.0;
        for (int j = 0; j < 19; j++)
            if (e[j]) acc = e[j] > 0 ? acc + f[j] : acc - f[j];
        if (a == 0 && it_pos) acc = acc + k.half_force;
        m.u[a] = acc / m.rho;
    }
    m.bad = m.rho > 1.2 || m.rho < 0.5;
    const double uv = (m.u[0] * m.u[0] + m.u[1] * m.u[1]) + m.u[2] * m.u[2];
    const double uv15 = 1.5 * uv;
    for (int j = 0; j < 19; j++) {
        double eu = 0.0;
        for (int a = 0; a < 3; a++)
            if (axis(a)[j]) eu = eu + (axis(a)[j] > 0 ? m.u[a] : -m.u[a]);
        const double feq =
            (ex_::wt(ex_::xc(j)) * m.rho) * (((1.0 + 3.0 * eu) + (4.5 * eu) * eu) - uv15);
        const double A = k.omega + (k.k3 * ((double)axis(0)[j] - m.u[0])) * k.force;
        f[j] = k.om1 * f[j] + A * feq;
    }
    return m;
}

double pick_tau(Rng &r, int mode)
{
    switch (mode) {
    case 0: return 0.55 + r.u();                              /* usual */
    case 1: return 1.0;                                       /* 1 - omega = 0 */
    case 2: return 1.0 + 0.06 * r.sym();                      /* small 1 - omega */
    case 3: return 1.0 + pow(10.0, -2.0 - 10.0 * r.u()) * (r.one_in(2) ? 1 : -1);
    case 4: return 0.5 + pow(10.0, -3.0 + 2.0 * r.u());       /* omega near 2 */
    default: return pow(10.0, 0.3 + 1.3 * r.u());             /* 2 to 40 */
    }
}

}  // namespace

/* n nodes of one kind of relaxation time; *inside receives how many lay in
 * the domain.  Returns the nodes whose bits differ. */
extern "C" long ex_check(long n, unsigned long long seed, int tau_mode, long *inside)
{
    Rng r{seed};
    long wrong = 0, in = 0;
    for (long t = 0; t < n; t++) {
        const double tau = pick_tau(r, tau_mode);
        double force = pow(10.0, -2.5 - 9.0 * r.u());
        if (r.one_in(12)) force = 0.0;
        if (r.one_in(8)) force = -force;
        const double om = 1.0 / tau;
        const ex_::Consts k =
            ex_::make_consts(om, 1.0 - om, (1.0 - 0.5 * om) * 3.0, force, 0.5 * force);
        /* near equilibrium at some density and velocity (each component up
         * to past the domain's 0.08), noise from none to 10%, now and then a
         * value at its weight, a short significand or a domain end */
        const double mag = pow(10.0, -0.9 - (r.one_in(3) ? 14.0 : 3.0) * r.u());
        const double rho = 1.0 + (r.one_in(4) ? 0.5 : 0.02) * (r.u() - 0.5);
        double U[3] = {mag * r.sym(), mag * r.sym(), mag * r.sym()};
        const uint64_t z = r.next() % 8;
        if (z < 3) U[z] = 0.0;
        if (z == 3) U[0] = U[1] = U[2] = 0.0;
        const double noise = r.one_in(5) ? 0.0 : pow(10.0, -(r.one_in(4) ? 1.0 : 3.0) - 14.0 * r.u());
        double f[19];
        uint64_t b[19], out[19] = {0};
        for (int j = 0; j < 19; j++) {
            const double w = ex_::wt(ex_::xc(j));
            double eu = 0.0, uu = 0.0;
            for (int a = 0; a < 3; a++) {
                eu += axis(a)[j] * U[a];
                uu += U[a] * U[a];
            }
            f[j] = w * rho * (1.0 + 3.0 * eu + 4.5 * eu * eu - 1.5 * uu) * (1.0 + noise * r.sym());
            if (r.one_in(64)) f[j] = w;
            if (r.one_in(512)) f[j] = w * (r.one_in(2) ? 0.29 : 1.68);
            b[j] = ex_::bits_of(f[j]);
            if (r.one_in(32)) b[j] &= ~((1ull << (r.next() % 52)) - 1ull);
            if (r.one_in(4000)) b[j] = r.next();
            f[j] = ex_::of_bits(b[j]);
        }
        const bool it_pos = r.one_in(2);
        ex_::Out o;
        auto store = [&](int j, uint64_t v) { out[j] = v; };
        uint32_t outside = 1u;
        if (k.ok == 1u) outside = ex_::collide<false>(b, k, it_pos, o, store);
        else if (k.ok == 2u) outside = ex_::collide<true>(b, k, it_pos, o, store);
        if (outside) continue;
        in++;
        const Macro m = reference(f, k, it_pos);
        bool same = o.rho == m.rho && o.u == m.u[0] && o.v == m.u[1] && o.w == m.u[2] &&
                    (o.bad != 0u) == m.bad;
        for (int j = 0; j < 19; j++) same = same && out[j] == ex_::bits_of(f[j]);
        wrong += !same;
    }
    *inside = in;
    return wrong;
}

/* rounded products at the ends of mulr's range against 128-bit integers */
extern "C" long mulr_check(long n, unsigned long long seed)
{
    Rng r{seed};
    long wrong = 0;
    for (long t = 0; t < n; t++) {
        uint64_t a = (r.next() | (1ull << 63)) >> (r.next() % 4);
        uint64_t c = (r.next() | (1ull << 63)) >> (r.next() % 6);
        if (r.one_in(3)) a &= ~0ull << (r.next() % 40);
        if (r.one_in(3)) c &= ~0ull << (r.next() % 40);
        if (r.one_in(50)) a = ~0ull >> 1;
        const unsigned __int128 p = (unsigned __int128)a * c;
        const uint64_t top = (uint64_t)(p >> 64);
        if ((a >> 32) + (c >> 32) >= (1ull << 32) || top < (1ull << 54) || top >> 63) continue;
        int d = 0;
        while ((top >> d) >> 53) d++;
        const unsigned __int128 half = (unsigned __int128)1 << (63 + d);
        unsigned __int128 q = p >> (64 + d);
        const unsigned __int128 rem = p - (q << (64 + d));
        if (rem > half || (rem == half && (q & 1))) q++;
        wrong += ex_::mulr(a, c) != ((uint64_t)q << d);
    }
    return wrong;
}
