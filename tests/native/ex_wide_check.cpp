/* The integer bit-exact collision (plb_ex.h) at large relaxation times, and
 * the moments it leaves for a node that is outside by its velocity, against
 * the same operations in the host's FP64, bit for bit. */
#include "ex_check.cpp"

namespace {

struct Node {
    double f[19];
    uint64_t b[19];
};

/* near equilibrium at velocity components up to `umax`, some noise */
Node make_node(Rng &r, double umax)
{
    Node n;
    double U[3], uu = 0.0;
    for (double &x : U) {
        x = umax * r.sym();
        if (r.one_in(8)) x = 0.0;
        if (umax > 0.1 && r.one_in(4)) x = (0.11 - 1e-3 * r.u() * r.u()) * (r.one_in(2) ? 1 : -1);
        uu += x * x;
    }
    const double rho = r.one_in(6) ? 0.5 + 0.72 * r.u() : 1.0 + 0.02 * (r.u() - 0.5);
    const double noise = r.one_in(5) ? 0.0 : pow(10.0, -(r.one_in(4) ? 1.5 : 3.0) - 14.0 * r.u());
    for (int j = 0; j < 19; j++) {
        double eu = 0.0;
        for (int a = 0; a < 3; a++) eu += axis(a)[j] * U[a];
        const double w = ex_::wt(ex_::xc(j));
        n.f[j] = w * rho * (1.0 + 3.0 * eu + 4.5 * eu * eu - 1.5 * uu) * (1.0 + noise * r.sym());
        if (r.one_in(64)) n.f[j] = w;
        n.b[j] = ex_::bits_of(n.f[j]);
        if (r.one_in(32)) n.b[j] &= ~((1ull << (r.next() % 52)) - 1ull);
        n.f[j] = ex_::of_bits(n.b[j]);
    }
    return n;
}

}  // namespace

/* rounded products from 2^117 on against 128-bit integers */
extern "C" long mulr_low_check(long n, unsigned long long seed)
{
    Rng r{seed};
    long wrong = 0;
    for (long t = 0; t < n; t++) {
        const uint64_t a = ((r.next() | (1ull << 63)) >> 4) & (~0ull << (r.next() % 50));
        const uint64_t c = ((r.next() | (1ull << 63)) >> (4 + r.next() % 3)) &
                           (~0ull << (r.next() % 50));
        const unsigned __int128 p = (unsigned __int128)a * c;
        const uint64_t top = (uint64_t)(p >> 64);
        if (top < (1ull << 53)) continue;
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

/* n nodes at tau in [lo, hi) and forces of magnitude up to fmax; *inside
 * receives those in the domain, *fast those outside by their velocity.
 * Returns the nodes whose values or moments differ. */
extern "C" long ex_wide_check(long n, unsigned long long seed, double lo, double hi, double fmax,
                              double umax, long *inside, long *fast)
{
    Rng r{seed};
    long wrong = 0, in = 0, quick = 0;
    for (long t = 0; t < n; t++) {
        const double tau = lo * pow(hi / lo, r.u());
        double force = fmax * pow(10.0, -9.0 * r.u()) * (r.one_in(8) ? -1.0 : 1.0);
        if (r.one_in(12)) force = 0.0;
        const double om = 1.0 / tau;
        const ex_::Consts k =
            ex_::make_consts(om, 1.0 - om, (1.0 - 0.5 * om) * 3.0, force, 0.5 * force);
        Node nd = make_node(r, umax * pow(10.0, -(r.one_in(3) ? 8.0 : 1.0) * r.u()));
        const bool it_pos = r.one_in(2);
        uint64_t out[19] = {0};
        auto store = [&](int j, uint64_t v) { out[j] = v; };
        ex_::Out o;
        uint32_t outside = ex_::kOutside;
        if (k.ok == 1u) outside = ex_::collide<false>(nd.b, k, it_pos, o, store);
        else if (k.ok == 2u) outside = ex_::collide<true>(nd.b, k, it_pos, o, store);
        if (outside == ex_::kOutside) continue;
        const Macro m = reference(nd.f, k, it_pos);
        bool same = o.rho == m.rho && o.u == m.u[0] && o.v == m.u[1] && o.w == m.u[2] &&
                    (o.bad != 0u) == m.bad;
        if (outside == ex_::kFast) {
            quick++;
        } else {
            in++;
            for (int j = 0; j < 19; j++) same = same && out[j] == ex_::bits_of(nd.f[j]);
        }
        wrong += !same;
    }
    *inside = in;
    *fast = quick;
    return wrong;
}
