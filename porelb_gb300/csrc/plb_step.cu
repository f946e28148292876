/*
 * plb_step.cu - the fused pull-stream + BGK collide + body-force step.
 *
 * One thread per fluid node.  Thread i gathers its 19 post-stream values
 * through the neighbour words (the on-device image of the reference's push
 * stream, stream_inner_nodes porelb.c:285-300), relaxes them (collision,
 * porelb.c:318-365) and writes its 19 post-collision values to the other
 * ping-pong buffer.  Distributions are SoA, f[j][npad], so the 19 stores and
 * the five neighbour-word loads of a warp (three of short words) are fully
 * coalesced; the gathers hit nodes that the row or Morton order keeps close in
 * memory.  On domains
 * larger than the L2 each CTA also asks L2 for the node range of a block some
 * way ahead (prefetch_block, prefetch_ctas).
 *
 * Forms:
 *   FP64_EXACT  the reference's operations in the reference's order with
 *               one rounding each: bit-exact.  Most of them run on the
 *               integer pipes (plb_ex.h), the rest and the nodes outside its
 *               domain with round-to-nearest intrinsics.
 *   FP64        exact Q60 fixed-point collision on the integer pipes
 *               (plb_fx.h); nodes outside its range fall back to FP64_FMA.
 *   FP64_FMA    the same algebra in native FP64, restructured for FMA.
 *   FP32/FP16DEV/BF16DEV  relative deviations g = f/w - 1 stored (scaled)
 *               in 32/16/16 bits, collision in FP32 on the deviations.
 */
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <string.h>

#include "plb_emu.h"
#include "plb_ex.h"
#include "plb_internal.h"

namespace plb {

/* weights of the three classes, as the reference's doubles (porelb.h:36-42) */
__device__ __forceinline__ double w64(int c)
{
    return c == 0 ? 1.0 / 3 : (c == 1 ? 1.0 / 18 : 1.0 / 36);
}
__device__ __forceinline__ float w32(int c)
{
    return c == 0 ? (float)(1.0 / 3) : (c == 1 ? (float)(1.0 / 18) : (float)(1.0 / 36));
}

__device__ __forceinline__ double dadd(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double dsub(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ double dmul(double a, double b) { return __dmul_rn(a, b); }
/* the same product on the integer pipes (plb_emu.h): the same bits for a
 * node whose values, density and run constants passed the range check.
 * The bit-exact collision outside plb_ex.h's domain sends 84 of its 97
 * products per node here, which balances the FP64 and integer pipes (2.05 ->
 * 2.68 GLUPS at 256^3); a node outside this range too takes the NATIVE
 * products. */
template <bool NATIVE>
__device__ __forceinline__ double imul(double a, double b)
{
    if constexpr (NATIVE) {
        return __dmul_rn(a, b);
    } else {
        return __longlong_as_double((long long)emu::dmul_bits_fast(
            (uint64_t)__double_as_longlong(a), (uint64_t)__double_as_longlong(b)));
    }
}

/* ------------------------------------------------------------- gather */

/* A step's launch overlaps the one before it (programmatic dependent
 * launch): its CTAs start while the last wave of the previous step drains,
 * read what no step writes (the neighbour words, the block maps) and then
 * wait for the previous grid to complete and its stores to be visible.  So
 * nothing before pdl_wait() may read distributions or write anything, and
 * the distributions, which the previous grid may still be writing when this
 * one starts, are read with plain loads, not through the read-only path. */
__device__ __forceinline__ void pdl_launch_next()
{
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
__device__ __forceinline__ void pdl_wait(bool launch)
{
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if (launch) pdl_launch_next();
}

/* A kernel's share of the rule in step_trigger.  Only the FP32 and 16-bit
 * forms' kernels for short launches can trigger after their gathers: the
 * trigger is a point that no load is moved across, and one that does not even
 * run costs the FP64 pool 5% and FP32 at 96^3 10%.  Where a kernel's launches
 * all take one place it is fixed (a choice costs the 16-bit forms 2-4%): the
 * start in these forms' long launches, after the gathers in the 16-bit forms'
 * short ones outside pools. */
template <int PREC, int W, bool POOL> struct TriggerPlace {
    static constexpr bool half = PREC == PLB_FP16DEV || PREC == PLB_BF16DEV;
    static constexpr bool dev = half || PREC == PLB_FP32;
    static constexpr bool early = dev && (W == kWordsLate || (W == kWordsShort && !POOL));
    static constexpr bool late = dev && W == kWordsFirst;
    static constexpr bool fixed_late = late && half && !POOL;
    static __device__ __forceinline__ void start(int t)
    {
        if (early || (!fixed_late && t == kTriggerStart)) pdl_launch_next();
    }
    static __device__ __forceinline__ bool waited(int t)
    {
        return !early && !fixed_late &&
               (t == kTriggerWaited || (!late && t == kTriggerGathered));
    }
    static __device__ __forceinline__ void gathered(int t)
    {
        if (fixed_late || (late && t == kTriggerGathered)) pdl_launch_next();
    }
};

/* word_at() for the form that stores T (FP32 alone has short words) */
template <typename T>
__device__ __forceinline__ long long word_place(int j, long long i, long long np)
{
    if constexpr (sizeof(T) == 4) return word_in_block(j, i);
    return word_in_rows(j, i, np);
}

template <typename T>
__device__ __forceinline__ void load_words(const uint32_t *nbr, long long np, long long i,
                                           int (&w)[Q - 1])
{
#pragma unroll
    for (int q = 0; q < 4; q++) {
        const int4 v = __ldg((const int4 *)(nbr + word_place<T>(4 * q + 1, i, np)));
        w[4 * q] = v.x;
        w[4 * q + 1] = v.y;
        w[4 * q + 2] = v.z;
        w[4 * q + 3] = v.w;
    }
    const int2 v = __ldg((const int2 *)(nbr + word_place<T>(17, i, np)));
    w[16] = v.x;
    w[17] = v.y;
}

template <typename T>
__device__ __forceinline__ void gather_words(const T *fin, long long np, long long i,
                                             const int (&w)[Q - 1], T (&f)[Q])
{
    f[0] = fin[i];
#pragma unroll
    for (int j = 1; j < Q; j++) f[j] = fin[(long long)j * np + w[j - 1]];
}

/* the same two in one: each gather waits for its own words alone */
template <typename T>
__device__ __forceinline__ void gather(const T *fin, const uint32_t *nbr,
                                       long long np, long long i, T (&f)[Q])
{
    int w[Q - 1];
    load_words<T>(nbr, np, i, w);
    gather_words<T>(fin, np, i, w, f);
}

/* The streamed values of node i (if valid), after the step before: WF loads
 * the neighbour words before the wait, else they are loaded after it and each
 * gather waits for its own (words_first_waves); `launch` triggers the next step's
 * launch after the wait. */
template <typename T, bool WF>
__device__ __forceinline__ void stream_node(const void *fin, const uint32_t *nbr,
                                            long long np, long long i, bool valid, bool launch,
                                            T (&f)[Q])
{
    if constexpr (WF) {
        int w[Q - 1];
        if (valid) load_words<T>(nbr, np, i, w);
        pdl_wait(launch);
        if (valid) gather_words<T>((const T *)fin, np, i, w, f);
    } else {
        pdl_wait(launch);
        if (valid) gather<T>((const T *)fin, nbr, np, i, f);
    }
}

/* the streamed values of node i from its short words q */
template <typename T>
__device__ __forceinline__ void gather_short(const T *fin, const uint32_t (&q)[9], long long np,
                                             long long i, int2 base, int rest, T (&f)[Q])
{
    f[0] = fin[i];
#pragma unroll
    for (int j = 1; j < Q; j++)
        f[j] = fin[(long long)j * np + short_word(q, j, (int)i, np, base, rest)];
}

/* ------------------------------------------------- FP64, reference order */

/* e.u as the reference evaluates ((e0*u + e1*v) + e2*w) (porelb.c:9): terms
 * with a zero coefficient add a signed zero, which changes no result. */
template <int J>
__device__ __forceinline__ double eu_ref(double u, double v, double w)
{
    double acc = 0.0;
    bool first = true;
    if (ex(J) != 0) { acc = ex(J) > 0 ? u : -u; first = false; }
    if (ey(J) != 0) {
        const double t = ey(J) > 0 ? v : -v;
        acc = first ? t : dadd(acc, t);
        first = false;
    }
    if (ez(J) != 0) {
        const double t = ez(J) > 0 ? w : -w;
        acc = first ? t : dadd(acc, t);
        first = false;
    }
    return acc;
}

/* rho_u etc. accumulated in j order (porelb.c:330-336).  The first nonzero
 * term is added to 0.0, which is exact. */
template <int C>
__device__ __forceinline__ double moment_ref(const double (&f)[Q])
{
    double acc = 0.0;
    bool first = true;
#pragma unroll
    for (int j = 0; j < Q; j++) {
        const int e = C == 0 ? ex(j) : (C == 1 ? ey(j) : ez(j));
        if (e == 0) continue;
        if (first) {
            acc = e > 0 ? f[j] : -f[j];
            first = false;
        } else {
            acc = e > 0 ? dadd(acc, f[j]) : dsub(acc, f[j]);
        }
    }
    return acc;
}

struct Macro {
    double rho, u, v, w;
    bool bad;
};

/* The collision from a node's moments (u shifted by the force): f(j) gives
 * the streamed values, store(j, x) takes the others.  Which products run on the
 * FP64 pipe: EQ those of the equilibrium, RELAX those of the relaxation. */
template <bool EQ, bool RELAX, typename Value, typename Store>
__device__ __forceinline__ void relax_fp64_exact(const Coeffs &a, double rho, double u, double v,
                                                 double w, const Value &f, const Store &store)
{
    const double uv = dadd(dadd(dmul(u, u), dmul(v, v)), dmul(w, w));
    const double uv15 = dmul(1.5, uv);
    const double h0 = dmul(w64(0), rho);
    const double h1 = dmul(w64(1), rho);
    const double h2 = dmul(w64(2), rho);
    /* omega + ((1-omega/2)*3*(e_x - u))*F for e_x = -1, 0, +1 */
    const double am = dadd(a.omega, dmul(dmul(a.k3, dsub(-1.0, u)), a.force));
    const double a0 = dadd(a.omega, dmul(dmul(a.k3, dsub(0.0, u)), a.force));
    const double ap = dadd(a.omega, dmul(dmul(a.k3, dsub(1.0, u)), a.force));

    /* rest direction: e.u = 0 gives ((1 + 0) + 0) - 1.5 uv */
    {
        const double feq = imul<EQ>(h0, dsub(1.0, uv15));
        store(0, dadd(imul<RELAX>(a.om1, f(0)), imul<RELAX>(a0, feq)));
    }
    /* pairs (J, J+1) with e_{J+1} = -e_J: 3 e.u, 4.5 e.u and (4.5 e.u) e.u
     * of the partner are exact negations / the same value. */
#pragma unroll
    for (int J = 1; J < Q; J += 2) {
        const int K = J + 1;
        const double eu = (J == 1) ? eu_ref<1>(u, v, w)
                        : (J == 3) ? eu_ref<3>(u, v, w)
                        : (J == 5) ? eu_ref<5>(u, v, w)
                        : (J == 7) ? eu_ref<7>(u, v, w)
                        : (J == 9) ? eu_ref<9>(u, v, w)
                        : (J == 11) ? eu_ref<11>(u, v, w)
                        : (J == 13) ? eu_ref<13>(u, v, w)
                        : (J == 15) ? eu_ref<15>(u, v, w)
                                    : eu_ref<17>(u, v, w);
        const double t3 = imul<EQ>(3.0, eu);
        const double c2 = imul<EQ>(imul<EQ>(4.5, eu), eu);
        const double h = wclass(J) == 1 ? h1 : h2;
        const double feqJ = imul<EQ>(h, dsub(dadd(dadd(1.0, t3), c2), uv15));
        const double feqK = imul<EQ>(h, dsub(dadd(dsub(1.0, t3), c2), uv15));
        const double AJ = ex(J) > 0 ? ap : (ex(J) < 0 ? am : a0);
        const double AK = ex(K) > 0 ? ap : (ex(K) < 0 ? am : a0);
        store(J, dadd(imul<RELAX>(a.om1, f(J)), imul<RELAX>(AJ, feqJ)));
        store(K, dadd(imul<RELAX>(a.om1, f(K)), imul<RELAX>(AK, feqK)));
    }
}

template <bool NATIVE>
__device__ __forceinline__ Macro collide_fp64_exact(double (&f)[Q],
                                                     const Coeffs &a, uint32_t &outside)
{
    Macro m;
    double rho = f[0];
#pragma unroll
    for (int j = 1; j < Q; j++) rho = dadd(rho, f[j]);
    double ru = moment_ref<0>(f);
    const double rv = moment_ref<1>(f);
    const double rw = moment_ref<2>(f);
    m.bad = (rho > 1.2) | (rho < 0.5);
    if constexpr (!NATIVE) {
        /* the density in [2^-64, 2^64) too, or the node takes the native
         * multiply (the caller) */
        const uint64_t rb = (uint64_t)__double_as_longlong(rho);
        outside |= emu::outside_node_range(rb) | (uint32_t)((rb << 1) == 0ull);
        if (outside) return m;
    }
    if (a.it > 0) ru = dadd(ru, a.half_force);
    m.rho = rho;
    m.u = __ddiv_rn(ru, rho);
    m.v = __ddiv_rn(rv, rho);
    m.w = __ddiv_rn(rw, rho);
    relax_fp64_exact<NATIVE, NATIVE>(a, rho, m.u, m.v, m.w, [&](int j) { return f[j]; },
                                     [&](int j, double x) { f[j] = x; });
    return m;
}

/* ------------------------------------------------------ FP64 with FMA */

__device__ __forceinline__ Macro collide_fp64_fma(double (&f)[Q],
                                                   const Coeffs &a)
{
    Macro m;
    double s[Q], d[Q];
#pragma unroll
    for (int J = 1; J < Q; J += 2) {
        s[J] = f[J] + f[J + 1];
        d[J] = f[J] - f[J + 1];
    }
    double rho = f[0];
#pragma unroll
    for (int J = 1; J < Q; J += 2) rho += s[J];
    double jx = 0.0, jy = 0.0, jz = 0.0;
#pragma unroll
    for (int J = 1; J < Q; J += 2) {
        if (ex(J)) jx += ex(J) * d[J];
        if (ey(J)) jy += ey(J) * d[J];
        if (ez(J)) jz += ez(J) * d[J];
    }
    m.bad = (rho > 1.2) | (rho < 0.5);
    if (a.it > 0) jx += a.half_force;
    const double inv = 1.0 / rho;
    const double u = jx * inv, v = jy * inv, w = jz * inv;
    m.rho = rho; m.u = u; m.v = v; m.w = w;
    const double uv15 = 1.5 * (u * u + v * v + w * w);
    const double c = a.k3 * a.force;
    const double am = a.omega - c * (1.0 + u);
    const double a0 = a.omega - c * u;
    const double ap = a.omega + c * (1.0 - u);
    const double h0 = w64(0) * rho, h1 = w64(1) * rho, h2 = w64(2) * rho;
    const double b1 = h1 - h1 * uv15, b2 = h2 - h2 * uv15;
    f[0] = a.om1 * f[0] + a0 * (h0 - h0 * uv15);
#pragma unroll
    for (int J = 1; J < Q; J += 2) {
        const int K = J + 1;
        const double eu = ex(J) * u + ey(J) * v + ez(J) * w;
        const double h = wclass(J) == 1 ? h1 : h2;
        const double b = wclass(J) == 1 ? b1 : b2;
        const double sym = fma(4.5 * h * eu, eu, b);
        const double anti = 3.0 * h * eu;
        const double AJ = ex(J) > 0 ? ap : (ex(J) < 0 ? am : a0);
        const double AK = ex(K) > 0 ? ap : (ex(K) < 0 ? am : a0);
        f[J] = fma(a.om1, f[J], AJ * (sym + anti));
        f[K] = fma(a.om1, f[K], AK * (sym - anti));
    }
    return m;
}

/* ----------------------------------------- FP32 collision on deviations */

/* g_j = f_j / w_j - 1.  With rho = 1 + delta, the BGK + force update
 *   f' = (1-omega) f + (omega + a_j) w rho (1 + P_j),
 *   a_j = 3 (1 - omega/2) F (e_jx - u),  P_j = 3 e.u + 4.5 (e.u)^2 - 1.5 u.u
 * becomes, exactly in real arithmetic,
 *   g'_j = (1-omega) g_j + omega delta + rho ((omega + a_j) P_j + a_j),
 * which keeps every FP32 quantity at deviation scale. */
__device__ __forceinline__ Macro collide_dev32(float (&g)[Q], const Coeffs &a)
{
    Macro m;
    float d[Q];
#pragma unroll
    for (int j = 0; j < Q; j++) d[j] = w32(wclass(j)) * g[j];
    float s[Q], df[Q];
#pragma unroll
    for (int J = 1; J < Q; J += 2) {
        s[J] = d[J] + d[J + 1];
        df[J] = d[J] - d[J + 1];
    }
    float delta = d[0];
#pragma unroll
    for (int J = 1; J < Q; J += 2) delta += s[J];
    float jx = 0.f, jy = 0.f, jz = 0.f;
#pragma unroll
    for (int J = 1; J < Q; J += 2) {
        if (ex(J)) jx += ex(J) * df[J];
        if (ey(J)) jy += ey(J) * df[J];
        if (ez(J)) jz += ez(J) * df[J];
    }
    const float rho = 1.0f + delta;
    m.bad = (rho > 1.2f) | (rho < 0.5f);
    if (a.it > 0) jx += a.half_force_f;
    const float inv = 1.0f / rho;
    const float u = jx * inv, v = jy * inv, w = jz * inv;
    m.rho = 1.0 + (double)delta;
    m.u = u; m.v = v; m.w = w;
    const float om = a.omega_f, om1 = a.om1_f;
    const float c = a.c_f;
    const float uv15 = 1.5f * (u * u + v * v + w * w);
    const float base = om * delta;
    const float am = -c * (1.0f + u), a0 = -c * u, ap = c * (1.0f - u);
    {
        const float P = -uv15;
        g[0] = fmaf(om1, g[0], base + rho * fmaf(om + a0, P, a0));
    }
#pragma unroll
    for (int J = 1; J < Q; J += 2) {
        const int K = J + 1;
        const float eu = ex(J) * u + ey(J) * v + ez(J) * w;
        const float sym = fmaf(4.5f * eu, eu, -uv15);
        const float PJ = fmaf(3.0f, eu, sym);
        const float PK = fmaf(-3.0f, eu, sym);
        const float aJ = ex(J) > 0 ? ap : (ex(J) < 0 ? am : a0);
        const float aK = ex(K) > 0 ? ap : (ex(K) < 0 ? am : a0);
        g[J] = fmaf(om1, g[J], base + rho * fmaf(om + aJ, PJ, aJ));
        g[K] = fmaf(om1, g[K], base + rho * fmaf(om + aK, PK, aK));
    }
    return m;
}

/* storage conversion of the deviation forms */
__device__ __forceinline__ float to_f(float x) { return x; }
__device__ __forceinline__ float to_f(__half x) { return __half2float(x); }
__device__ __forceinline__ float to_f(__nv_bfloat16 x) { return __bfloat162float(x); }
template <typename T> __device__ __forceinline__ T from_f(float x);
template <> __device__ __forceinline__ float from_f<float>(float x) { return x; }
template <> __device__ __forceinline__ __half from_f<__half>(float x) { return __float2half_rn(x); }
template <> __device__ __forceinline__ __nv_bfloat16 from_f<__nv_bfloat16>(float x) { return __float2bfloat16_rn(x); }

/* --------------------------------------------------------------- kernel */

/* ----------------------------------------- FP64 on the integer pipes */

template <bool MACRO, typename Store>
__device__ __forceinline__ Macro collide_fx(const double (&f)[Q], const Coeffs &a,
                                            bool &fallback, const Store &store)
{
    uint64_t b[Q];
#pragma unroll
    for (int j = 0; j < Q; j++) b[j] = (uint64_t)__double_as_longlong(f[j]);
    fx::Moments mm;
    const uint32_t fl = fx::collide(b, a.fxk, a.it > 0, mm, store);
    Macro m;
    fallback = (fl & fx::kBad) != 0;
    m.bad = (fl & fx::kDensity) != 0;
    if (MACRO) {
        uint32_t ignore = 0;
        m.rho = __longlong_as_double((long long)fx::to_bits(mm.R, ignore));
        m.u = (double)fx::mul(mm.Jx, mm.inv) * 0x1p-60;
        m.v = (double)fx::mul(mm.Jy, mm.inv) * 0x1p-60;
        m.w = (double)fx::mul(mm.Jz, mm.inv) * 0x1p-60;
    } else {
        m.rho = m.u = m.v = m.w = 0.0;
    }
    return m;
}

template <int PREC> struct StoreOf { using T = double; };
template <> struct StoreOf<PLB_FP32> { using T = float; };
template <> struct StoreOf<PLB_FP16DEV> { using T = __half; };
template <> struct StoreOf<PLB_BF16DEV> { using T = __nv_bfloat16; };

/* Largest CTA (T) and resident CTAs of that size per SM (v) the register
 * budget is set for, by kernel variant (0 = default; 1 and 3 the
 * alternatives the launch tuner tries).
 * Fixed-point FP64: 5 x 128 threads, 96 registers (322 us at 256^3, 1258 at
 * 400^3; 128 registers 330 and 1368, 80 registers 333 and 1300: fewer warps
 * wait longer, tighter budgets spill); 256-thread CTAs on request (V = 4) 128
 * registers; the alternatives 80 and 64.
 * FP32 and 16-bit forms: 48 registers (FP16 39.1 GLUPS at 512^3 against 38.4
 * unconstrained) or, with the words held before the wait, 64 (at 48 they
 * spill: FP16 at 92k nodes 2.94 against 2.75 us); the alternatives
 * unconstrained and 40.
 * Bit-exact FP64: 80 (its integer chains wait on themselves, so warps pay:
 * 5.9 GLUPS at 256^3 against 4.9 with 108 registers and 16 warps per SM; 64
 * registers spill: 5.7).  FMA FP64: unconstrained. */
template <int PREC, int V, int W> struct MinBlocks {
    static constexpr bool dev = PREC == PLB_FP32 || PREC == PLB_FP16DEV || PREC == PLB_BF16DEV;
    static constexpr int T = PREC == PLB_FP64 && V == 0 ? 128 : 256;
    static constexpr int v = PREC == PLB_FP64 ? (V == 1 ? 3 : V == 3 ? 4 : V == 4 ? 2 : 5)
                           : dev ? (V == 1 ? 1 : V == 3 ? 6 : W == kWordsFirst ? 4 : 5)
                         : PREC == PLB_FP64_EXACT ? 3 : 1;
    /* for the batch step's CTAs of BT threads */
    static constexpr int batch(int BT)
    {
        return PREC == PLB_FP64 ? (BT == 128 ? 5 : 2) : v * (kBatchBlock / BT);
    }
};

/* The bit-exact collision of node i that left plb_ex.h's domain by its
 * velocity, from its moments: its streamed values, gathered again, are needed
 * one by one, and all 19 are stored again (128^3 with half or all of the nodes
 * past the range: 449 and 480 us a step; from the values alone 662 and 635;
 * with the equilibrium's products on the integer pipes too 522 and 503, with
 * none there 440 and 531).  Out of line, so the common path keeps its
 * registers. */
__device__ __noinline__ void exact_node_fast(const double *fin, double *fout, const uint32_t *nbr,
                                             long long np, long long i, const Coeffs *run,
                                             double rho, double u, double v, double w)
{
    int at[Q - 1];
    load_words<double>(nbr, np, i, at);
    auto value = [&](int j) { return fin[j == 0 ? i : (long long)j * np + at[j - 1]]; };
    auto store = [&](int j, double x) { __stcs(fout + (long long)j * np + i, x); };
    if (run->exact_native) relax_fp64_exact<true, true>(*run, rho, u, v, w, value, store);
    else relax_fp64_exact<true, false>(*run, rho, u, v, w, value, store);
}

/* The bit-exact collision of node i outside plb_ex.h's common domain, from
 * its streamed values gathered again, stored: plb_ex.h's form for tau within
 * 1/16 of 1 or above 32 (128^3: 192 us a step, the products' form 358); else
 * the products on the integer pipes for a node in their range, every product
 * on the FP64 pipe for one whose values or density (or the run's constants)
 * lie outside it, such as an infinity, a NaN, a subnormal or an extreme value.
 * Out of line, so the common path keeps its registers. */
__device__ __noinline__ Macro exact_node_wide(const double *fin, double *fout,
                                              const uint32_t *nbr, long long np,
                                              long long i, const Coeffs *run, int it,
                                              unsigned int *flags)
{
    Coeffs co = *run;
    co.it = it;
    double raw[Q];
    gather<double>(fin, nbr, np, i, raw);
    Macro m;
    uint32_t outside = co.exk.ok ^ 2u;
    if (!outside) {
        uint64_t b[Q];
#pragma unroll
        for (int j = 0; j < Q; j++) b[j] = (uint64_t)__double_as_longlong(raw[j]);
        ex_::Out o;
        outside = ex_::collide<true>(b, co.exk, co.it > 0, o, [&](int j, uint64_t v) {
            __stcs(fout + (long long)j * np + i, __longlong_as_double((long long)v));
        });
        if (outside == ex_::kFast) {
            exact_node_fast(fin, fout, nbr, np, i, run, o.rho, o.u, o.v, o.w);
            if (co.exact_native) *flags |= 2u;
        }
        if (outside != ex_::kOutside) {
            m.rho = o.rho; m.u = o.u; m.v = o.v; m.w = o.w;
            m.bad = o.bad != 0u;
            return m;
        }
    }
    /* the integer multiply needs the node's values in [2^-64, 2^64) (and its
     * density, checked in the collision): their smallest and largest exponent
     * field (a zero value, which the range admits but a distribution never
     * is, takes the native path) */
    uint32_t emin = 0x7ffu, emax = 0u;
#pragma unroll
    for (int j = 0; j < Q; j++) {
        const uint32_t e = ((uint32_t)__double2hiint(raw[j]) >> 20) & 0x7ffu;
        emin = min(emin, e);
        emax = max(emax, e);
    }
    outside = (uint32_t)co.exact_native | (uint32_t)(emin < 1023u - 64u) |
              (uint32_t)(emax > 1023u + 63u);
    if (!outside) m = collide_fp64_exact<false>(raw, co, outside);
    if (outside) {
        *flags |= 2u;
        gather<double>(fin, nbr, np, i, raw);
        uint32_t unused = 0;
        m = collide_fp64_exact<true>(raw, co, unused);
    }
#pragma unroll
    for (int j = 0; j < Q; j++) __stcs(fout + (long long)j * np + i, raw[j]);
    return m;
}

/* Collide node i's streamed values raw[] and store them.  run: co in global
 * or parameter memory (its iteration number may be another's), for the path
 * that is out of line. */
template <int PREC, bool MACRO, typename T>
__device__ __forceinline__ Macro collide_node(T (&raw)[Q], const T *fin, T *fout,
                                              const uint32_t *nbr, long long np,
                                              long long i, const Coeffs &co,
                                              const Coeffs *run, unsigned int &flags,
                                              float &dev_max)
{
    Macro m;
    if constexpr (PREC == PLB_FP64) {
        bool fallback;
        m = collide_fx<MACRO>(raw, co, fallback, [&](int j, uint64_t v) {
            __stcs(fout + (long long)j * np + i, __longlong_as_double((long long)v));
        });
        if (fallback) {
            /* outside the fixed-point range: native FP64 from the streamed
             * values, gathered again, all 19 stored again */
            gather<T>(fin, nbr, np, i, raw);
            m = collide_fp64_fma(raw, co);
            flags |= 2u;
#pragma unroll
            for (int j = 0; j < Q; j++) __stcs(fout + (long long)j * np + i, raw[j]);
        }
    } else if constexpr (PREC == PLB_FP64_EXACT) {
        uint64_t b[Q];
#pragma unroll
        for (int j = 0; j < Q; j++) b[j] = (uint64_t)__double_as_longlong(raw[j]);
        ex_::Out o;
        uint32_t outside = co.exk.ok == 1u ? 0u : ex_::kOutside;
        if (!outside)
            outside = ex_::collide<false>(b, co.exk, co.it > 0, o, [&](int j, uint64_t v) {
                __stcs(fout + (long long)j * np + i, __longlong_as_double((long long)v));
            });
        /* these store all 19 values again */
        if (outside == ex_::kOutside)
            return exact_node_wide(fin, fout, nbr, np, i, run, co.it, &flags);
        if (outside == ex_::kFast) {
            exact_node_fast(fin, fout, nbr, np, i, run, o.rho, o.u, o.v, o.w);
            if (co.exact_native) flags |= 2u;
        }
        m.rho = o.rho; m.u = o.u; m.v = o.v; m.w = o.w;
        m.bad = o.bad != 0u;
    } else if constexpr (PREC == PLB_FP64_FMA) {
        m = collide_fp64_fma(raw, co);
#pragma unroll
        for (int j = 0; j < Q; j++) __stcs(fout + (long long)j * np + i, raw[j]);
    } else {
        float g[Q];
#pragma unroll
        for (int j = 0; j < Q; j++) g[j] = to_f(raw[j]) * co.inv_scale;
        m = collide_dev32(g, co);
        float big = 0.f;
#pragma unroll
        for (int j = 0; j < Q; j++) {
            const float h = g[j] * co.scale;
            big = fmaxf(big, fabsf(h));
            fout[(long long)j * np + i] = from_f<T>(h);
        }
        if (PREC == PLB_FP16DEV && !(big <= 60000.f)) flags |= 1u;
        dev_max = big;
    }
    return m;
}

/* Bulk L2 prefetch of [p, p + bytes), bytes a positive multiple of 16 and
 * p 16-byte aligned. */
__device__ __forceinline__ void prefetch_l2(const void *p, unsigned bytes)
{
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(bytes) : "memory");
}

/* Thread 0 of a block asks L2 for the node range of block b (a block that
 * starts some time after this one, pf_blocks blocks later in launch order):
 * its rows of neighbour words and its 19 rows of distributions.  In
 * Morton order most gathers of that block read inside the ranges of the
 * blocks launched near it, so its loads then wait for L2 instead of DRAM.
 * Rows are npad elements (a multiple of 64) and the block size is a multiple
 * of 32, so every range starts 64-byte aligned and spans a multiple of 64
 * bytes inside its row or its word block. */
template <typename T>
__device__ __forceinline__ void prefetch_block(const T *fin, const uint32_t *nbr,
                                               const int2 *shorts, long long np, long long n,
                                               long long b, int bs)
{
    const long long i0 = b * bs;
    if (i0 >= n) return;
    const long long cnt = np - i0 < bs ? np - i0 : bs;
    const unsigned fb = (unsigned)(cnt * (long long)sizeof(T));
    /* one range or, where the words of 256 nodes lie together, one for each
     * such block that this one touches */
    for (long long k = i0; k < i0 + cnt;) {
        long long end = i0 + cnt;
        if (sizeof(T) == 4 && (k | 255) + 1 < end) end = (k | 255) + 1;
        const unsigned m = (unsigned)(end - k);
        if (shorts && shorts[k >> 8].x != kWholeWords) {
            const uint32_t *p = nbr + (k >> 8) * kWordBlock;
            prefetch_l2(p + 4 * (k & 255), m * 16);
            prefetch_l2(p + 1024 + 4 * (k & 255), m * 16);
            prefetch_l2(p + 2048 + (k & 255), m * 4);
        } else {
#pragma unroll 1
            for (int j = 1; j < 17; j += 4) prefetch_l2(nbr + word_place<T>(j, k, np), m * 16);
            prefetch_l2(nbr + word_place<T>(17, k, np), m * 8);
        }
        k = end;
    }
#pragma unroll 1
    for (int j = 0; j < Q; j++) prefetch_l2(fin + (long long)j * np + i0, fb);
}

template <int PREC, bool MACRO, int VARIANT, int W>
__global__ void
__launch_bounds__((MinBlocks<PREC, VARIANT, W>::T), (MinBlocks<PREC, VARIANT, W>::v))
k_step(const StepArgs a)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (a.pf_blocks > 0 && threadIdx.x == 0)
        prefetch_block<typename StoreOf<PREC>::T>((const typename StoreOf<PREC>::T *)a.fin,
                                                  a.nbr, W == kWordsShort ? a.shorts : nullptr,
                                                  a.npad, a.n,
                                                  (long long)blockIdx.x + a.pf_blocks,
                                                  blockDim.x);
    using T = typename StoreOf<PREC>::T;
    T raw[Q];
    using Trig = TriggerPlace<PREC, W, false>;
    const bool launch = Trig::waited(a.trigger);
    Trig::start(a.trigger);
    if constexpr (PREC == PLB_FP64) {
        /* one kernel for both, as fast as two (256^3 315.7 against 314.6 us,
         * 24^3 2.68 against 2.83); FP32 and 16-bit kernels are the ones with
         * registers to lose to a branch */
        if (a.words_first) stream_node<T, true>(a.fin, a.nbr, a.npad, i, i < a.n, launch, raw);
        else stream_node<T, false>(a.fin, a.nbr, a.npad, i, i < a.n, launch, raw);
    } else if constexpr (W == kWordsShort) {
        /* the short words are asked for before it is known whether the block
         * has them: a block that has not (1 in 60) reads 36 bytes a node
         * for nothing, the others wait for one load less */
        uint32_t q[9];
        int2 base = make_int2(0, 0);
        if (i < a.n) {
            load_short(a.nbr, i, q);
            base = __ldg(a.shorts + (i >> 8));
        }
        pdl_wait(launch);
        if (i < a.n) {
            if (base.x != kWholeWords) gather_short<T>((const T *)a.fin, q, a.npad, i, base, a.n, raw);
            else gather<T>((const T *)a.fin, a.nbr, a.npad, i, raw);
        }
    } else {
        stream_node<T, W == kWordsFirst>(a.fin, a.nbr, a.npad, i, i < a.n, launch, raw);
    }
    Trig::gathered(a.trigger);
    double sum_u = 0.0, sum_r = 0.0;
    if (i < a.n) {
        float dm = 0.f;
        unsigned int fl = 0;
        const Macro m = collide_node<PREC, MACRO>(raw, (const T *)a.fin, (T *)a.fout, a.nbr,
                                                  a.npad, i, a.co, &a.co, fl, dm);
        if (fl) atomicOr(a.flags, fl);
        if (m.bad) {
            const unsigned long long key =
                ((unsigned long long)(unsigned)a.co.it << 32) | (unsigned)a.perm[i];
            atomicMin(a.err, key);
        }
        if (MACRO) {
            const long long np = a.npad;
            a.macro[i] = m.rho;
            a.macro[np + i] = m.u;
            a.macro[2 * np + i] = m.v;
            a.macro[3 * np + i] = m.w;
            sum_u = m.u;
            sum_r = m.rho;
        }
    }
    if (MACRO) {
        __shared__ double su[32], sr[32];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            sum_u += __shfl_down_sync(0xffffffffu, sum_u, o);
            sum_r += __shfl_down_sync(0xffffffffu, sum_r, o);
        }
        const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
        if (lane == 0) { su[wid] = sum_u; sr[wid] = sum_r; }
        __syncthreads();
        if (threadIdx.x == 0) {
            double tu = 0.0, tr = 0.0;
            for (int k = 0; k < (int)(blockDim.x >> 5); k++) { tu += su[k]; tr += sr[k]; }
            a.partial[blockIdx.x] = tu;
            a.partial[gridDim.x + blockIdx.x] = tr;
        }
    }
}

/* Batch step: kBatchBlock / BT CTAs of BT threads per active pool block;
 * CTA b works on part b % H of pool block blk_list[b / H] (of the current
 * L2 group's window of the list, when the pool steps in groups), whose map
 * entry blk_sample[] packs its sample and that sample's node count in it.  CTAs
 * that run at the same time work on neighbouring pool blocks, so in Morton
 * order their gathers share L2 lines (a fixed grid looping over the list
 * lost that and ran 23% slower in the FP64 form). */
template <int PREC, bool MACRO, int BT, int W>
__global__ void __launch_bounds__(BT, (MinBlocks<PREC, 0, W>::batch(BT)))
k_batch_step(const BatchArgs a)
{
    using T = typename StoreOf<PREC>::T;
    constexpr int H = kBatchBlock / BT; /* CTAs per pool block */
    const int *list = a.blk_list;
    int ncta = (int)gridDim.x;
    if (a.grp) {
        /* one L2 group of the interval: its window of the block list */
        const int g = *a.grp_cur;
        list += a.grp[2 * g];
        ncta = a.grp[2 * g + 1] * H;
        if ((int)blockIdx.x >= ncta) return;
    }
    const int part = blockIdx.x % H;
    const int pb = list[blockIdx.x / H];
    const int packed = a.blk_sample[pb];
    const int s = packed >> 9;                  /* -1: free block */
    const int k = part * BT + threadIdx.x;      /* node within the pool block */
    const bool valid = s >= 0 && k < (packed & 511);
    const long long i = (long long)pb * kBatchBlock + k;
    /* L2 prefetch of the part of a pool block the CTA pf_blocks later steps */
    if (a.pf_blocks > 0 && threadIdx.x == 0 && (int)blockIdx.x + a.pf_blocks < ncta) {
        const unsigned c = blockIdx.x + a.pf_blocks;
        prefetch_block<T>((const T *)a.fin, a.nbr, W == kWordsShort ? a.shorts : nullptr,
                          a.npad, a.npad,
                          (long long)list[c / H] * H + c % H, BT);
    }
    double sum_u = 0.0, sum_r = 0.0;
    float dmax = 0.f;
    /* the gathers first: they need only the node's place in the pool.  The
     * block maps and words above and below are the interval's: no step
     * writes them, so they are read before the wait (see k_step) */
    T raw[Q];
    using Trig = TriggerPlace<PREC, W, true>;
    const bool launch = Trig::waited(a.trigger);
    Trig::start(a.trigger);
    int2 base = make_int2(kWholeWords, 0);
    if (W == kWordsShort) base.x = a.shorts[pb].x;
    if (W == kWordsShort && base.x != kWholeWords) {
        uint32_t q[9];
        if (valid) {
            load_short(a.nbr, i, q);
            base.y = a.shorts[pb].y; /* (with x in one load: 3% at 92k nodes) */
        }
        pdl_wait(launch);
        if (valid) gather_short<T>((const T *)a.fin, q, a.npad, i, base, a.rest, raw);
    } else {
        stream_node<T, W == kWordsFirst>(a.fin, a.nbr, a.npad, i, valid, launch, raw);
    }
    Trig::gathered(a.trigger);
    if (valid) {
        {
            /* the sample's coefficients straight from global memory (the
             * same record for the whole CTA: cached after the first warp);
             * no shared-memory staging, so no barrier makes the warps wait
             * for each other's gathers */
            const SampleDev *sp = a.samples + s;
            Coeffs co = sp->co;
            co.it = *a.t_base + a.t_off - sp->start;
            unsigned int fl = 0;
            const Macro m = collide_node<PREC, MACRO>(raw, (const T *)a.fin, (T *)a.fout,
                                                      a.nbr, a.npad, i, co, &sp->co, fl, dmax);
            if (fl | (m.bad ? 4u : 0u)) atomicOr(a.serr + s, fl | (m.bad ? 4u : 0u));
            if (MACRO) {
                const long long np = a.npad;
                if (a.macro) {
                    a.macro[i] = m.rho;
                    a.macro[np + i] = m.u;
                    a.macro[2 * np + i] = m.v;
                    a.macro[3 * np + i] = m.w;
                }
                sum_u = m.u;
                sum_r = m.rho;
            }
        }
    }
    if (MACRO) {
        __shared__ double su[32], sr[32];
        __shared__ float sd[32];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            sum_u += __shfl_down_sync(0xffffffffu, sum_u, o);
            sum_r += __shfl_down_sync(0xffffffffu, sum_r, o);
            dmax = fmaxf(dmax, __shfl_down_sync(0xffffffffu, dmax, o));
        }
        const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
        if (lane == 0) { su[wid] = sum_u; sr[wid] = sum_r; sd[wid] = dmax; }
        __syncthreads();
        if (threadIdx.x == 0) {
            double tu = 0.0, tr = 0.0;
            float td = 0.f;
            for (int w = 0; w < BT / 32; w++) {
                tu += su[w];
                tr += sr[w];
                td = fmaxf(td, sd[w]);
            }
            const long long row = (long long)pb * H + part;
            a.partial[row] = tu;
            a.partial[a.part_stride + row] = tr;
            a.partial[2 * a.part_stride + row] = (double)td;
        }
    }
}

/* One step launch, overlapping the kernel before it in the stream (see
 * pdl_wait). */
static cudaError_t launch_pdl(void (*fn)(StepArgs), int grid, int block, const StepArgs &a,
                              cudaStream_t s)
{
    cudaLaunchConfig_t c;
    memset(&c, 0, sizeof(c));
    c.gridDim = dim3((unsigned)grid);
    c.blockDim = dim3((unsigned)block);
    c.stream = s;
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    c.attrs = &at;
    c.numAttrs = 1;
    return cudaLaunchKernelEx(&c, fn, a);
}

template <int PREC, int V>
static void (*step_fn(bool macros, int words))(StepArgs)
{
    if constexpr (short_form(PREC))
        if (words == kWordsShort)
            return macros ? k_step<PREC, true, V, kWordsShort> : k_step<PREC, false, V, kWordsShort>;
    if constexpr (PREC != PLB_FP64)
        if (words == kWordsFirst)
            return macros ? k_step<PREC, true, V, kWordsFirst> : k_step<PREC, false, V, kWordsFirst>;
    return macros ? k_step<PREC, true, V, kWordsLate> : k_step<PREC, false, V, kWordsLate>;
}

/* the tighter register budgets are built for the tuned forms only */
template <int PREC>
static void (*step_variant(bool macros, int words, int variant))(StepArgs)
{
    if constexpr (PREC == PLB_FP64 || PREC == PLB_FP32 || PREC == PLB_FP16DEV ||
                  PREC == PLB_BF16DEV) {
        if (variant == 1) return step_fn<PREC, 1>(macros, words);
        if (variant == 3) return step_fn<PREC, 3>(macros, words);
    }
    if constexpr (PREC == PLB_FP64)
        if (variant == 4) return step_fn<PREC, 4>(macros, words);
    return step_fn<PREC, 0>(macros, words);
}

template <int PREC>
static cudaError_t launch_prec(bool macros, const StepArgs &a, const StepLaunch &l,
                               cudaStream_t s)
{
    const int grid = (a.n + l.block - 1) / l.block;
    if (grid == 0) return cudaSuccess;
    return launch_pdl(step_variant<PREC>(macros, l.words, l.variant), grid, l.block, a, s);
}

/* CTAs of a kernel resident on an SM of the current device, and its SMs;
 * false if unknown. */
static bool occupancy(const void *fn, int block, int *per, int *sms)
{
    int dev = 0;
    return cudaGetDevice(&dev) == cudaSuccess &&
           cudaDeviceGetAttribute(sms, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess &&
           cudaOccupancyMaxActiveBlocksPerMultiprocessor(per, fn, block, 0) == cudaSuccess;
}

/* Where a step of `grid` CTAs of `block` threads, `per` of them to an SM,
 * lets the next step's CTAs start: at once where the launch fills the device.
 * In a shorter one the CTAs of the steps after would pile up on the SMs that
 * are free first, several of one step on an SM and none on others, and a step
 * take up to twice its time (FMA form at 46k nodes 30 against 20 us, FP64 at
 * 38k 6.1 against 3.8, FP32 at 39k 3.3 against 2.2).  There
 *   FP32, 16-bit  after the gathers (FP32 at 92k nodes 3.0 us, right after the
 *                 wait 3.8); in a pool of few CTAs, which reads its block maps
 *                 first, right after the wait (FP16, 76k nodes: 2.6 / 3.4)
 *   FP64 forms    right after the wait while an SM has a CTA or two; more of
 *                 them keep it busy for long enough that the next step's have
 *                 to find it free: at this step's end (bit-exact at 61k nodes
 *                 17.7 us, after the wait 23.5; FP64 at 22k 4.1 / 3.7)
 * An alternative, CTAs that ask for so much shared memory that an SM holds no
 * more than its share, is as fast (92k nodes FP32 3.3 us, FP16 2.75) but keeps
 * other handles off the device: eight FP32 handles of 92k nodes then take 43
 * us for a step each, and 28 without. */
static int step_trigger(int precision, bool pool, long long grid, int block, int per, int sms)
{
    const long long share = (grid + sms - 1) / sms; /* CTAs of an SM */
    if (precision == PLB_FP64_EXACT || precision == PLB_FP64 || precision == PLB_FP64_FMA) {
        if (share > per) return kTriggerStart;
        const long long few = precision == PLB_FP64_FMA ? 128 : 256; /* threads */
        return grid * block > few * sms && share < per ? kTriggerExit : kTriggerWaited;
    }
    if (share >= per) return kTriggerStart;
    return pool && share <= 3 && share * block <= 512 ? kTriggerWaited : kTriggerGathered;
}

/* L2 bytes of the current device, 0 if unknown */
static int l2_bytes()
{
    int dev = 0, l2 = 0;
    return cudaGetDevice(&dev) == cudaSuccess &&
                   cudaDeviceGetAttribute(&l2, cudaDevAttrL2CacheSize, dev) == cudaSuccess
               ? l2 : 0;
}

/* L2 prefetch distance in CTAs for a launch over `nodes` nodes, `wave` CTAs
 * resident at once; want: 1 on, -1 off, 0 where it pays, which is once what a
 * step moves outgrows the L2 (96^3 FP64, in L2: 22.3 us without, 23.2 with).
 * Distances in 32nds of a wave, the fastest of 1 to 32:
 *   plain step   FP64 8 (256^3: none 359 us, 8 318, 16 322), 16-bit 12 (FP16
 *                none 141, 8 131, 12 129), FP32 6 with short words (none 166,
 *                4 163, 6 163, 16 166); with wide ones FP32 loses (none 190,
 *                8 193)
 *   pool step    FP64 12 (16 x 96^3: none 334, 8 301, 12 294, 16 296), FP32 16
 *                with short words (none 141, 8 142, 16 139) and 8 without (none
 *                162, 8 157, 24 163), 16-bit 16 (none 124, 8 114, 16 110) */
int prefetch_ctas(int precision, long long nodes, int wave, bool pool, bool shorts, int want)
{
    const bool fp64 = precision == PLB_FP64;
    const bool half = precision == PLB_FP16DEV || precision == PLB_BF16DEV;
    const bool fp32 = precision == PLB_FP32;
    if (want < 0) return 0;
    if (want == 0) {
        if (!fp64 && !half && !(fp32 && (pool || shorts))) return 0;
        const int l2 = l2_bytes();
        if (l2 <= 0 || nodes * (2 * Q * (fp64 ? 8 : fp32 ? 4 : 2) + (shorts ? 36 : 72)) <= l2)
            return 0;
    }
    const int part = half  ? (pool ? 16 : 12)
                     : fp64 ? (pool ? 12 : 8)
                     : pool ? (shorts ? 16 : 8)
                            : (shorts ? 6 : 8);
    return (wave * part + 31) / 32;
}

/* Short words cost a step about 100 instructions a node and save it 36 of 224
 * bytes of DRAM traffic, so they are for node sets that outgrow the L2
 * (FP32, wide then short: 96^3 6.7 and 8.1 us, 108^3 12.5 and 11.3, 128^3
 * 25.3 and 22.0, 256^3 190 and 166, 400^3 715 and 627).  The line lies
 * at two thirds of it (393k nodes; 108^3 has 441k).  The 16-bit forms are
 * not bound by DRAM (256^3 FP16 with short words 137 us, with wide 129) and
 * neither are the FP64 ones (327 and 318). */
bool short_words_pay(int precision, long long nodes)
{
    return short_form(precision) && l2_bytes() > 0 &&
           nodes * (2 * Q * 4 + 72) > l2_bytes() / 3 * 2;
}

template <int PREC>
static void plan_prec(int n, StepLaunch *l)
{
    int per = 0, sms = 0;
    const int grid = (n + l->block - 1) / l->block;
    /* blocks of the (non-macro) kernel resident on the whole device at once:
     * the unit of the L2 prefetch distance */
    l->wave = occupancy((const void *)step_variant<PREC>(false, kWordsLate, l->variant), l->block,
                        &per, &sms) ? sms * per : 0;
    l->words = grid <= words_first_waves(PREC) * (long long)l->wave ? kWordsFirst : kWordsLate;
    l->trigger = occupancy((const void *)step_variant<PREC>(false, l->words, l->variant), l->block,
                           &per, &sms) ? step_trigger(PREC, false, grid, l->block, per, sms)
                                       : kTriggerStart;
}

void plan_step(int precision, int n, StepLaunch *l)
{
    switch (precision) {
    case PLB_FP64_EXACT: return plan_prec<PLB_FP64_EXACT>(n, l);
    case PLB_FP64: return plan_prec<PLB_FP64>(n, l);
    case PLB_FP64_FMA: return plan_prec<PLB_FP64_FMA>(n, l);
    case PLB_FP32: return plan_prec<PLB_FP32>(n, l);
    case PLB_FP16DEV: return plan_prec<PLB_FP16DEV>(n, l);
    case PLB_BF16DEV: return plan_prec<PLB_BF16DEV>(n, l);
    default: return;
    }
}

/* Threads per CTA of the plain step.  128 for the fixed-point and FMA FP64
 * forms (FP64 at 256^3 319 us, with 256 threads 366); 256 for the others once
 * 128-thread CTAs fill the device (bit-exact form 990 against 1101 us at
 * 256^3, FP16 130 / 135), and 128 below, where the finer grain spreads better
 * (at 92k nodes bit-exact 20.7 against 23.4 us, FP32 3.0 / 3.3).  Domains that
 * 64-thread CTAs cover with one per SM take those: fewer warps share an SM's
 * pipes (4.6k nodes: FMA 6.8 against 7.5 us, FP64 2.62 / 2.71, bit-exact 8.6 /
 * 8.5). */
template <int PREC>
static int block_prec(int n)
{
    int per = 0, sms = 0;
    if (!occupancy((const void *)step_variant<PREC>(false, false, 0), 128, &per, &sms)) return 256;
    if (n <= sms * 64) return 64;
    if (PREC == PLB_FP64 || PREC == PLB_FP64_FMA) return 128;
    return n <= (long long)sms * per * 128 ? 128 : 256;
}

int step_block(int precision, int n)
{
    switch (precision) {
    case PLB_FP64_EXACT: return block_prec<PLB_FP64_EXACT>(n);
    case PLB_FP64: return block_prec<PLB_FP64>(n);
    case PLB_FP64_FMA: return block_prec<PLB_FP64_FMA>(n);
    case PLB_FP32: return block_prec<PLB_FP32>(n);
    case PLB_FP16DEV: return block_prec<PLB_FP16DEV>(n);
    case PLB_BF16DEV: return block_prec<PLB_BF16DEV>(n);
    default: return 256;
    }
}

/* Threads per CTA of the batch step by default: 128 for the fixed-point
 * FP64 form (two CTAs per pool block; 4% faster in the plain kernel), 256
 * otherwise.  A pool may choose either (the launch tuner times both). */
int batch_default_cta(int precision)
{
    return precision == PLB_FP64 ? 128 : kBatchBlock;
}

template <int PREC, int BT>
static int batch_wave_bt()
{
    int per = 0, sms = 0;
    return occupancy((const void *)k_batch_step<PREC, false, BT, kWordsFirst>, BT, &per, &sms) ? sms * per
                                                                                      : 0;
}

template <int PREC>
static int batch_wave_prec(int cta)
{
    return cta == 128 ? batch_wave_bt<PREC, 128>() : batch_wave_bt<PREC, kBatchBlock>();
}

int batch_wave_blocks(int precision, int cta)
{
    switch (precision) {
    case PLB_FP64_EXACT: return batch_wave_prec<PLB_FP64_EXACT>(cta);
    case PLB_FP64: return batch_wave_prec<PLB_FP64>(cta);
    case PLB_FP64_FMA: return batch_wave_prec<PLB_FP64_FMA>(cta);
    case PLB_FP32: return batch_wave_prec<PLB_FP32>(cta);
    case PLB_FP16DEV: return batch_wave_prec<PLB_FP16DEV>(cta);
    case PLB_BF16DEV: return batch_wave_prec<PLB_BF16DEV>(cta);
    default: return 0;
    }
}

template <int PREC, int BT>
static const void *batch_fn(bool macros, int words)
{
    if constexpr (short_form(PREC)) {
        if (words == kWordsShort)
            return macros ? (const void *)k_batch_step<PREC, true, BT, kWordsShort>
                          : (const void *)k_batch_step<PREC, false, BT, kWordsShort>;
    }
    if constexpr (MinBlocks<PREC, 0, kWordsFirst>::dev) {
        if (words == kWordsLate)
            return macros ? (const void *)k_batch_step<PREC, true, BT, kWordsLate>
                          : (const void *)k_batch_step<PREC, false, BT, kWordsLate>;
    }
    return macros ? (const void *)k_batch_step<PREC, true, BT, kWordsFirst>
                  : (const void *)k_batch_step<PREC, false, BT, kWordsFirst>;
}

/* The pool's words come first in every launch of the FP64 forms (0.1M to 6M
 * nodes: 3-6% faster than words after the wait); the deviation forms', up to
 * the same number of waves as a plain step's (FP32 92k nodes 3.6 against 3.9
 * us, 5M nodes 171 against 162).  A pool with short words reads them first:
 * nine registers hold them (5M nodes 138 us). */
template <int PREC>
static const void *batch_fn_cta(bool macros, int cta, int grid, bool shorts)
{
    const int words = shorts ? kWordsShort
                      : grid <= (long long)words_first_waves(PREC) * batch_wave_prec<PREC>(cta)
                          ? kWordsFirst : kWordsLate;
    return cta == 128 ? batch_fn<PREC, 128>(macros, words)
                      : batch_fn<PREC, kBatchBlock>(macros, words);
}

const void *batch_step_kernel(int precision, bool macros, int cta, int grid, bool shorts)
{
    if (cta != 128 && cta != kBatchBlock) return nullptr;
    switch (precision) {
    case PLB_FP64_EXACT: return batch_fn_cta<PLB_FP64_EXACT>(macros, cta, grid, shorts);
    case PLB_FP64: return batch_fn_cta<PLB_FP64>(macros, cta, grid, shorts);
    case PLB_FP64_FMA: return batch_fn_cta<PLB_FP64_FMA>(macros, cta, grid, shorts);
    case PLB_FP32: return batch_fn_cta<PLB_FP32>(macros, cta, grid, shorts);
    case PLB_FP16DEV: return batch_fn_cta<PLB_FP16DEV>(macros, cta, grid, shorts);
    case PLB_BF16DEV: return batch_fn_cta<PLB_BF16DEV>(macros, cta, grid, shorts);
    default: return nullptr;
    }
}

int batch_step_trigger(int precision, int cta, int grid, bool shorts)
{
    int per = 0, sms = 0;
    const void *fn = batch_step_kernel(precision, false, cta, grid, shorts);
    return fn && occupancy(fn, cta, &per, &sms) ? step_trigger(precision, true, grid, cta, per, sms)
                                                : kTriggerStart;
}

cudaError_t launch_step(int precision, bool macros, const StepArgs &a, const StepLaunch &l,
                        cudaStream_t s)
{
    switch (precision) {
    case PLB_FP64_EXACT: return launch_prec<PLB_FP64_EXACT>(macros, a, l, s);
    case PLB_FP64: return launch_prec<PLB_FP64>(macros, a, l, s);
    case PLB_FP64_FMA: return launch_prec<PLB_FP64_FMA>(macros, a, l, s);
    case PLB_FP32: return launch_prec<PLB_FP32>(macros, a, l, s);
    case PLB_FP16DEV: return launch_prec<PLB_FP16DEV>(macros, a, l, s);
    case PLB_BF16DEV: return launch_prec<PLB_BF16DEV>(macros, a, l, s);
    default: return cudaErrorInvalidValue;
    }
}

}  // namespace plb
