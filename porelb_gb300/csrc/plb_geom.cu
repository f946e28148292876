/*
 * plb_geom.cu - device-side geometry: the periodic sphere-pack generator and
 * the node table built straight from a flag grid.
 *
 * build_V (preprocess.c:29-164) numbers fluid cells (flag == 1) in x-fastest
 * lexicographic order and stores, per node, the 18 neighbours at x + e_j.
 * From a flag grid the same information is a bit test: here the fluid cells
 * are ranked twice with popcount scans over bitmaps - once in lexicographic
 * order (the reference node number, used for the dump order and for the
 * order-dependent bounce-back rule) and once along the Morton curve (the
 * device order) - and the pull table is written directly, without the
 * 152-byte-per-node V.bin records.  For a flag with values 0/1 the result is
 * identical to plb_create on the table plb_build_table writes.
 */
#include <math.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include "plb_internal.h"

namespace plb {

/* ------------------------------------------------------------- bitmaps */

/* bits 0..3: the four 0/1 bytes of v */
__device__ __forceinline__ uint32_t nibble(uint32_t v)
{
    return (v * 0x01020408u) >> 24 & 15u;
}

/* lexicographic fluid bitmap: word w covers cells 32w .. 32w+31 (flag is 16-
 * byte aligned) */
__global__ void k_flag_bits(const uint8_t *flag, size_t cells, uint32_t *bits,
                            uint32_t *cnt, size_t words, unsigned *bad)
{
    const size_t w = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (w >= words) return;
    uint32_t b = 0, over = 0;
    const size_t c0 = w * 32;
    if (c0 + 32 <= cells) {
#pragma unroll
        for (int q = 0; q < 2; q++) {
            const uint4 v = __ldg((const uint4 *)(flag + c0) + q);
            over |= v.x | v.y | v.z | v.w;
            b |= (nibble(v.x) | nibble(v.y) << 4 | nibble(v.z) << 8 | nibble(v.w) << 12)
                 << (16 * q);
        }
    } else {
        for (int k = 0; k < (int)(cells - c0); k++) {
            over |= flag[c0 + k];
            b |= (uint32_t)(flag[c0 + k] & 1u) << k;
        }
    }
    if (over & 0xfefefefeu) atomicOr(bad, 1u);
    bits[w] = b;
    cnt[w] = __popc(b);
}

__device__ __forceinline__ uint32_t rank_in(const uint32_t *bits,
                                            const uint32_t *offs, uint64_t c)
{
    const uint32_t w = bits[c >> 5];
    return offs[c >> 5] + __popc(w & ((1u << (c & 31)) - 1u));
}

__device__ __forceinline__ bool bit_at(const uint32_t *bits, uint64_t c)
{
    return (bits[c >> 5] >> (c & 31)) & 1u;
}

__host__ __device__ inline uint64_t morton_code(uint32_t x, uint32_t y,
                                                uint32_t z, int bx, int by,
                                                int bz)
{
    uint64_t c = 0;
    int pos = 0;
    const int top = bx > by ? (bx > bz ? bx : bz) : (by > bz ? by : bz);
    for (int k = 0; k < top; k++) {
        if (k < bx) c |= (uint64_t)((x >> k) & 1u) << pos++;
        if (k < by) c |= (uint64_t)((y >> k) & 1u) << pos++;
        if (k < bz) c |= (uint64_t)((z >> k) & 1u) << pos++;
    }
    return c;
}

struct Grid {
    int nx, ny, nz;
    int bx, by, bz;
    int morton; /* 0 = device order is the reference order */
};

__device__ __forceinline__ uint64_t device_key(const Grid &g, int x, int y, int z)
{
    return morton_code(x, y, z, g.bx, g.by, g.bz);
}

__global__ void k_mark_order(const uint32_t *lexbits, Grid g, size_t cells,
                             uint32_t *obits)
{
    const size_t c = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= cells || !bit_at(lexbits, c)) return;
    const int x = (int)(c % g.nx);
    const int y = (int)((c / g.nx) % g.ny);
    const int z = (int)(c / ((size_t)g.nx * g.ny));
    const uint64_t k = device_key(g, x, y, z);
    atomicOr(obits + (k >> 5), 1u << (k & 31));
}

/* total fluid cells (meta[0]; meta[1] is the bad-value flag) and the first
 * node of every z slab (meta[2 ..]) */
__global__ void k_rank_meta(const uint32_t *bits, const uint32_t *offs, size_t words,
                            size_t cells, size_t slab_cells, int num_p, uint32_t *meta)
{
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p == 0) meta[0] = offs[words - 1] + __popc(bits[words - 1]);
    if (p < num_p) {
        const size_t c = (size_t)p * slab_cells;
        meta[2 + p] = c < cells ? rank_in(bits, offs, c)
                                : offs[words - 1] + __popc(bits[words - 1]);
    }
}

/* What the pull words of one node are made from and go to. */
struct TableArgs {
    const uint32_t *lexbits, *lexoffs; /* reference order */
    const uint32_t *obits, *ooffs;     /* device order (Morton) */
    Grid g;
    int slab, remote_wins, halfway, n;
    long long npad, rows;
    uint32_t word_base, rest_word;
    int *perm;
    uint16_t *coord;
    uint32_t *nbr;
};

/* Pull words of the node k on cell (x, y, z): see k_build_nbr for the rule.
 * s = x - e_j pushes into x if fluid; x bounces if t = x + e_j is solid; when
 * both write, the later in node order wins, i.e. the push iff s's cell index
 * is larger (lexicographic numbering is monotone in the cell index) - or
 * always when s lies in another rank slab and remote_wins is set.  Each of
 * the 18 neighbours is looked up once, for the direction it sends and the
 * one it stops. */
template <bool ROW>
__device__ __forceinline__ void node_words(const TableArgs &a, int x, int y, int z, size_t cx,
                                           long long k)
{
    const Grid &g = a.g;
    uint32_t idx[Q];
    uint32_t fluid = 0, later = 0, remote = 0;
    const int zs = a.remote_wins ? z / a.slab : 0;
#pragma unroll
    for (int j = 1; j < Q; j++) {
        int X = x + ex(j), Y = y + ey(j), Z = z + ez(j);
        X = X < 0 ? X + g.nx : (X >= g.nx ? X - g.nx : X);
        Y = Y < 0 ? Y + g.ny : (Y >= g.ny ? Y - g.ny : Y);
        Z = Z < 0 ? Z + g.nz : (Z >= g.nz ? Z - g.nz : Z);
        const size_t c = ((size_t)Z * g.ny + Y) * g.nx + X;
        const uint32_t w = __ldg(a.lexbits + (c >> 5)), bit = 1u << (c & 31);
        idx[j] = 0;
        if (w & bit) {
            fluid |= 1u << j;
            idx[j] = a.word_base + (ROW ? __ldg(a.lexoffs + (c >> 5)) + __popc(w & (bit - 1u))
                                        : rank_in(a.obits, a.ooffs, device_key(g, X, Y, Z)));
        }
        later |= (uint32_t)(c > cx) << j;
        if (a.remote_wins) remote |= (uint32_t)(Z / a.slab != zs) << j;
    }
    uint32_t words[Q - 1];
#pragma unroll
    for (int j = 1; j < Q; j++) {
        const int o = opp(j);
        const bool push = fluid >> o & 1u, bounce = !(fluid >> j & 1u);
        const bool wins = a.halfway || !bounce || ((later | remote) >> o & 1u);
        words[j - 1] = push && wins ? idx[o]
                     : a.halfway || bounce
                         ? bounce_word(j, (long long)a.word_base + k, a.npad)
                         : a.rest_word;
    }
    store_words(a.nbr, (long long)a.word_base + k, a.rows, words);
}

/* x, y, z of a cell */
__device__ __forceinline__ void cell_xyz(const Grid &g, size_t c, int &x, int &y, int &z)
{
    if (c >> 32) {
        x = (int)(c % g.nx);
        y = (int)((c / g.nx) % g.ny);
        z = (int)(c / ((size_t)g.nx * g.ny));
    } else {
        const uint32_t r = (uint32_t)c / (uint32_t)g.nx;
        x = (int)((uint32_t)c - r * (uint32_t)g.nx);
        z = (int)(r / (uint32_t)g.ny);
        y = (int)(r - (uint32_t)z * (uint32_t)g.ny);
    }
}

/* device index, reference index and coordinates of every fluid cell.  In row
 * order (ROW) the reference rank is the device index, and no second bitmap
 * is made. */
template <bool ROW>
__global__ void k_assign_from_flag(const TableArgs a, size_t cells)
{
    const size_t c = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= cells || !bit_at(a.lexbits, c)) return;
    int x, y, z;
    cell_xyz(a.g, c, x, y, z);
    const uint32_t i = rank_in(a.lexbits, a.lexoffs, c);
    const uint32_t k = ROW ? i : rank_in(a.obits, a.ooffs, device_key(a.g, x, y, z));
    if (k >= (uint32_t)a.n) return;
    a.perm[k] = (int)i;
    a.coord[k] = (uint16_t)x;
    a.coord[a.npad + k] = (uint16_t)y;
    a.coord[2 * a.npad + k] = (uint16_t)z;
}

/* pull table, a thread per node */
template <bool ROW>
__global__ void k_nbr_from_flag(const TableArgs a)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= a.n) return;
    const int x = a.coord[k], y = a.coord[a.npad + k], z = a.coord[2 * a.npad + k];
    node_words<ROW>(a, x, y, z, ((size_t)z * a.g.ny + y) * a.g.nx + x, k);
}

/* One CTA per block of 256 nodes; see shorten_words. */
__global__ void __launch_bounds__(kWordNodes)
k_shorten_words(uint32_t *nbr, int2 *shorts, long long lo, int n, int rest, int rewrite, int *count)
{
    __shared__ int least[3], most[3]; /* distances, by dz_planes() + 1 */
    const long long blk = (lo >> 8) + blockIdx.x;
    const long long i = blk * kWordNodes + threadIdx.x;
    if (threadIdx.x < 3) {
        least[threadIdx.x] = 0x7fffffff;
        most[threadIdx.x] = -0x7fffffff;
    }
    __syncthreads();
    int a[3] = {0x7fffffff, 0x7fffffff, 0x7fffffff};
    int b[3] = {-0x7fffffff, -0x7fffffff, -0x7fffffff};
    if (i < lo + n) {
#pragma unroll
        for (int j = 1; j < Q; j++) {
            const int s = (int)nbr[word_at(j, i, 0)];
            if (s == rest || s < lo || s >= lo + n) continue;
            const int d = s - (int)i, z = dz_planes(j) + 1;
            a[z] = min(a[z], d);
            b[z] = max(b[z], d);
        }
    }
#pragma unroll
    for (int z = 0; z < 3; z++) {
        const int l = __reduce_min_sync(0xffffffffu, a[z]), m = __reduce_max_sync(0xffffffffu, b[z]);
        if ((threadIdx.x & 31) == 0) {
            atomicMin(&least[z], l);
            atomicMax(&most[z], m);
        }
    }
    __syncthreads();
    /* those to another plane count from the smallest (none: from 0) */
    const int2 base = make_int2(least[2] > most[2] ? 0 : least[2],
                                least[0] > most[0] ? 0 : least[0]);
    constexpr int kMost = (int)kShortBounce - 1; /* the largest distance kept */
    const bool all = (least[2] > most[2] || most[2] - least[2] <= kMost) &&
                     (least[0] > most[0] || most[0] - least[0] <= kMost) &&
                     (least[1] > most[1] ||
                      (least[1] >= -kShortBias && most[1] <= kMost - kShortBias));
    if (threadIdx.x == 0) {
        shorts[blk] = all ? base : make_int2(kWholeWords, 0);
        if (all && count) atomicAdd(count, 1);
    }
    if (!all || !rewrite) return;
    uint32_t q[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
    if (i < lo + n) {
#pragma unroll
        for (int j = 1; j < Q; j++) {
            const int s = (int)nbr[word_at(j, i, 0)];
            uint32_t d = kShortBounce;
            if (s == rest) d = kShortRest;
            else if (s >= lo && s < lo + n)
                d = (uint32_t)(s - (int)i - (dz_planes(j) == 0  ? -kShortBias
                                             : dz_planes(j) > 0 ? base.x
                                                                : base.y));
            q[(j - 1) >> 1] |= d << ((j & 1) ? 0 : 16);
        }
    }
    /* every word of the block has been read when the first is rewritten */
    __syncthreads();
    uint32_t *p = nbr + blk * kWordBlock;
    ((uint4 *)p)[threadIdx.x] = make_uint4(q[0], q[1], q[2], q[3]);
    ((uint4 *)p)[256 + threadIdx.x] = make_uint4(q[4], q[5], q[6], q[7]);
    p[2048 + threadIdx.x] = q[8];
}

cudaError_t shorten_words(uint32_t *nbr, int2 *shorts, long long lo, int n, int rest,
                          bool rewrite, int *count, cudaStream_t st)
{
    if (n <= 0) return cudaSuccess;
    k_shorten_words<<<(unsigned)((n + kWordNodes - 1) / kWordNodes), kWordNodes, 0, st>>>(
        nbr, shorts, lo, n, rest, rewrite, count);
    return cudaGetLastError();
}

/* --------------------------------------------------------- sphere pack */

/* Same inside test as plb_sphere_pack (plb_host.c), with round-to-nearest
 * intrinsics so no FMA contraction changes a bit. */
__device__ __forceinline__ double min_image_d(double a, double c, int n)
{
    const double d = fabs(__dsub_rn(a, c));
    const double w = __dsub_rn((double)n, d);
    return d <= w ? d : w;
}

/* splitmix64 (Steele, Lea & Flood 2014), the same stream as plb_host.c: its
 * k-th draw needs no draw before it */
__device__ __forceinline__ double draw(uint64_t seed, uint64_t k)
{
    uint64_t z = seed + (k + 1) * 0x9E3779B97F4A7C15ULL;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ULL;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBULL;
    z ^= z >> 31;
    return __dmul_rn((double)(long long)(z >> 11), 0x1.0p-53);
}

/* cells along one axis that the tables hold: a wider bounding box is done in
 * parts of up to kBox^3 cells */
constexpr int kBox = 96;
constexpr int kCoverThreads = 128;

/* One block per sphere (blockIdx.x) and part of its bounding box (blockIdx.y
 * and every gridDim.y after it): every cell that lies inside takes the
 * sphere's index if it is the first to cover it.  The squared
 * distances along each axis are made once, in FP64 as the rule states, and
 * kept in shared memory; a warp takes a row of cells along x and decides them
 * in FP32 where the sum is clear of r^2 by more than FP32 can be off, in FP64
 * where it is not.  In FP64 alone, nine operations a cell, the FP64 pipe
 * bound the generator (200 x 192 x 210 cells, 18174 spheres: 2945 us, now
 * 316; 160^3 cells, spheres of radius 53 to 80: the whole call 27.7 ms, now
 * 3.1). */
__global__ void __launch_bounds__(kCoverThreads)
k_cover(uint64_t seed, long long base, int nx, int ny, int nz, double rmin, double rmax,
        uint32_t *first)
{
    __shared__ double d2[3][kBox];
    __shared__ float f2[3][kBox]; /* (a conversion is an FP64-pipe operation) */
    __shared__ int cell[3][kBox];
    const long long s = base + blockIdx.x;
    const uint32_t idx = (uint32_t)s;
    const int n[3] = {nx, ny, nz};
    const double c[3] = {__dmul_rn(draw(seed, 4 * s), (double)nx),
                         __dmul_rn(draw(seed, 4 * s + 1), (double)ny),
                         __dmul_rn(draw(seed, 4 * s + 2), (double)nz)};
    const double r = __dadd_rn(rmin, __dmul_rn(__dsub_rn(rmax, rmin), draw(seed, 4 * s + 3)));
    const double r2 = __dmul_rn(r, r);
    int lo[3], w[3], parts[3];
#pragma unroll
    for (int d = 0; d < 3; d++) {
        lo[d] = (int)floor(c[d] - r) - 1;
        int hi = (int)ceil(c[d] + r) + 1;
        if (hi - lo[d] + 1 > n[d]) hi = lo[d] + n[d] - 1;
        w[d] = hi - lo[d] + 1;
        parts[d] = (w[d] + kBox - 1) / kBox;
    }
    const long long all = (long long)parts[0] * parts[1] * parts[2];
    for (long long p = blockIdx.y; p < all; p += gridDim.y) {
        const int at[3] = {(int)(p % parts[0]) * kBox,
                           (int)(p / parts[0] % parts[1]) * kBox,
                           (int)(p / ((long long)parts[0] * parts[1])) * kBox};
        int m[3];
#pragma unroll
        for (int d = 0; d < 3; d++) {
            m[d] = min(w[d] - at[d], kBox);
            for (int t = threadIdx.x; t < m[d]; t += kCoverThreads) {
                const int q = (((lo[d] + at[d] + t) % n[d]) + n[d]) % n[d];
                const double e = min_image_d((double)q, c[d], n[d]);
                cell[d][t] = q;
                d2[d][t] = __dmul_rn(e, e);
                f2[d][t] = (float)d2[d][t];
            }
        }
        __syncthreads();
        /* FP32: each d2 and r2 rounded once, two adds: within 2^-22 */
        const float in = (float)r2 * (1.f - 1e-6f), out = (float)r2 * (1.f + 1e-6f);
        const int lane = threadIdx.x & 31;
        const int rows = m[1] * m[2];
        for (int row = threadIdx.x >> 5; row < rows; row += kCoverThreads / 32) {
            const int iz = row / m[1], iy = row - iz * m[1];
            const float dyz = f2[1][iy] + f2[2][iz];
            if (dyz > out) continue;
            uint32_t *const line = first + ((size_t)cell[2][iz] * ny + cell[1][iy]) * nx;
            for (int ix = lane; ix < m[0]; ix += 32) {
                const float e = f2[0][ix] + dyz;
                if (e > out) continue;
                if (e >= in &&
                    !(__dadd_rn(__dadd_rn(d2[0][ix], d2[1][iy]), d2[2][iz]) <= r2))
                    continue;
                uint32_t *const q = line + cell[0][ix];
                if (*(volatile uint32_t *)q > idx) atomicMin(q, idx);
            }
        }
        __syncthreads(); /* the tables are the next part's */
    }
}

/* hist[f - lo] += 1 for every cell first covered by sphere f in [lo, hi);
 * four cells a thread, runs of one sphere added at once */
__global__ void k_first_hist(const uint32_t *first, size_t cells, uint32_t lo,
                             uint32_t hi, unsigned long long *hist)
{
    const size_t c = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) * 4;
    if (c >= cells) return;
    uint32_t f[4];
    if (c + 4 <= cells) {
        const uint4 v = *(const uint4 *)(first + c);
        f[0] = v.x; f[1] = v.y; f[2] = v.z; f[3] = v.w;
    } else {
        for (int k = 0; k < 4; k++) f[k] = c + k < cells ? first[c + k] : hi;
    }
    uint32_t run = 0;
#pragma unroll
    for (int k = 0; k < 4; k++) {
        run++;
        if (k < 3 && f[k + 1] == f[k]) continue;
        if (f[k] >= lo && f[k] < hi) atomicAdd(hist + (f[k] - lo), (unsigned long long)run);
        run = 0;
    }
}

__global__ void k_popc_words(const uint32_t *bits, uint32_t *cnt, size_t m)
{
    const size_t k = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (k < m) cnt[k] = __popc(bits[k]);
}

__global__ void k_flag_from_first(const uint32_t *first, size_t cells,
                                  uint32_t nsph, uint8_t *flag)
{
    const size_t c = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) * 4;
    if (c + 4 <= cells) {
        const uint4 v = *(const uint4 *)(first + c);
        *(uchar4 *)(flag + c) = make_uchar4(v.x >= nsph, v.y >= nsph, v.z >= nsph, v.w >= nsph);
    } else {
        for (size_t k = c; k < cells; k++) flag[k] = first[k] < nsph ? 0 : 1;
    }
}

}  // namespace plb

using namespace plb;

/* ------------------------------------------------------ host interfaces */

namespace plb {

static unsigned gsz(size_t n, int b) { return (unsigned)((n + b - 1) / b); }

static int ceil_log2i(int v)
{
    int b = 0;
    while ((1LL << b) < v) b++;
    return b;
}

#define CKG(call)                                                             \
    do {                                                                      \
        cudaError_t e_ = (call);                                              \
        if (e_ != cudaSuccess) {                                              \
            fprintf(stderr, "porelb_gpu: %s failed: %s\n", #call,             \
                    cudaGetErrorString(e_));                                  \
            rc = e_ == cudaErrorMemoryAllocation ? PLB_ERR_NOMEM : PLB_ERR_CUDA; \
            goto done;                                                        \
        }                                                                     \
    } while (0)

/* Spheres drawn at a time: the expected count for the target porosity from
 * the mean volume, and a third more. */
static long long pack_chunk(size_t cells, double rmin, double rmax, double porosity)
{
    const double rm = 0.5 * (rmin + rmax);
    const double v = 4.18879020478639 * rm * rm * rm;
    const long long chunk =
        (long long)(-log(porosity > 1e-6 ? porosity : 1e-6) * (double)cells / v * 1.3) + 64;
    return chunk > 4000000 ? 4000000 : chunk;
}

/* Parts of the widest bounding box, for k_cover's grid. */
static unsigned cover_parts(int nx, int ny, int nz, double rmin, double rmax)
{
    const double wide = 2.0 * fmax(fabs(rmin), fabs(rmax)) + 6.0;
    double all = 1.0;
    for (int n : {nx, ny, nz}) all *= ceil(fmin(wide, (double)n) / kBox);
    return all < 65535.0 ? (unsigned)all : 65535u;
}

static size_t up256(size_t b) { return (b + 255) / 256 * 256; }

/* One device block for everything a geometry is made with. */
int geom_alloc(GeomWork *w, int nx, int ny, int nz, int num_p)
{
    const size_t cells = (size_t)nx * ny * nz;
    const size_t words = (cells + 31) / 32;
    const size_t lines = up256(words * 4);
    memset(w, 0, sizeof(*w));
    const size_t tmp = up256(scan_tmp_bytes(words));
    const size_t meta = up256(4 * ((size_t)num_p + 2));
    if (plb_cuda_malloc(&w->block, up256(cells) + 3 * lines + tmp + meta) != cudaSuccess)
        return PLB_ERR_NOMEM;
    char *p = w->block;
    w->flag = (uint8_t *)p;
    p += up256(cells);
    w->lexbits = (uint32_t *)p;
    p += lines;
    w->lexoffs = (uint32_t *)p;
    p += lines;
    w->cnt = (uint32_t *)p;
    p += lines;
    w->tmp = (uint32_t *)p;
    p += tmp;
    w->meta = (uint32_t *)p;
    return PLB_OK;
}

void geom_free(GeomWork *w)
{
    cudaFree(w->block);
    w->block = nullptr;
}

int sphere_pack_device(uint64_t seed, int nx, int ny, int nz, double rmin,
                       double rmax, double porosity, uint8_t *dflag,
                       int *num_spheres, double *porosity_out, cudaStream_t st)
{
    const size_t cells = (size_t)nx * ny * nz;
    const double total = (double)cells;
    int rc = PLB_OK;
    uint32_t *first = nullptr;
    unsigned long long *hist = nullptr;
    unsigned long long *hh = nullptr;
    char *block = nullptr;
    long long made = 0, ns = -1;
    long long fluid = (long long)cells;
    const long long chunk = pack_chunk(cells, rmin, rmax, porosity);
    const unsigned parts = cover_parts(nx, ny, nz, rmin, rmax);
    const size_t hbytes = sizeof(unsigned long long) * (size_t)chunk;
    CKG(plb_cuda_malloc(&block, up256(cells * 4) + hbytes));
    first = (uint32_t *)block;
    hist = (unsigned long long *)(block + up256(cells * 4));
    CKG(cudaMemsetAsync(first, 0xff, cells * 4, st));
    hh = (unsigned long long *)malloc(hbytes);
    if (!hh) { rc = PLB_ERR_NOMEM; goto done; }
    if (!((double)fluid / total > porosity)) ns = 0;
    while (ns < 0) {
        if (made > 100000000LL) { rc = PLB_ERR_ARG; goto done; }
        k_cover<<<dim3((unsigned)chunk, parts), kCoverThreads, 0, st>>>(seed, made, nx, ny, nz,
                                                                       rmin, rmax, first);
        CKG(cudaGetLastError());
        /* cells first covered by each sphere of this chunk */
        CKG(cudaMemsetAsync(hist, 0, hbytes, st));
        k_first_hist<<<gsz((cells + 3) / 4, 256), 256, 0, st>>>(first, cells, (uint32_t)made,
                                                               (uint32_t)(made + chunk), hist);
        CKG(cudaGetLastError());
        CKG(cudaMemcpyAsync(hh, hist, hbytes, cudaMemcpyDeviceToHost, st));
        CKG(cudaStreamSynchronize(st));
        for (long long k = 0; k < chunk && ns < 0; k++) {
            fluid -= (long long)hh[k];
            if (!((double)fluid / total > porosity)) ns = made + k + 1;
        }
        made += chunk;
        if (ns < 0 && made + chunk > 0x7fffffffLL) { rc = PLB_ERR_ARG; goto done; }
    }
    k_flag_from_first<<<gsz((cells + 3) / 4, 256), 256, 0, st>>>(first, cells, (uint32_t)ns,
                                                                dflag);
    CKG(cudaGetLastError());
    CKG(cudaStreamSynchronize(st));
    if (num_spheres) *num_spheres = (int)ns;
    if (porosity_out) *porosity_out = (double)fluid / total;
done:
    cudaStreamSynchronize(st);
    cudaFree(block);
    free(hh);
    return rc;
}

/* Lexicographic ranks of the fluid cells of w's flag grid: bitmap and word
 * offsets into w.  *n receives the fluid count, slab_start[num_p] the first
 * node of every z slab. */
int flag_rank(const GeomWork &w, int nx, int ny, int nz, int num_p, int *n, int *slab_start,
              cudaStream_t st)
{
    const size_t cells = (size_t)nx * ny * nz;
    const size_t words = (cells + 31) / 32;
    int rc = PLB_OK;
    uint32_t *h = (uint32_t *)malloc(4 * ((size_t)num_p + 2));
    if (!h) return PLB_ERR_NOMEM;
    CKG(cudaMemsetAsync(w.meta, 0, 8, st));
    k_flag_bits<<<gsz(words, 256), 256, 0, st>>>(w.flag, cells, w.lexbits, w.cnt, words,
                                                w.meta + 1);
    CKG(cudaGetLastError());
    rc = scan_words(w.cnt, w.lexoffs, words, w.tmp, st);
    if (rc != PLB_OK) goto done;
    k_rank_meta<<<gsz((size_t)num_p, 256), 256, 0, st>>>(w.lexbits, w.lexoffs, words, cells,
                                                        (size_t)(nz / num_p) * nx * ny, num_p,
                                                        w.meta);
    CKG(cudaGetLastError());
    CKG(cudaMemcpyAsync(h, w.meta, 4 * ((size_t)num_p + 2), cudaMemcpyDeviceToHost, st));
    CKG(cudaStreamSynchronize(st));
    if (h[1] || (long long)h[0] >= kMaxNodes) {
        rc = PLB_ERR_ARG;
        goto done;
    }
    *n = (int)h[0];
    for (int p = 0; p < num_p; p++) slab_start[p] = (int)h[2 + p];
done:
    free(h);
    return rc;
}

/* Morton (or reference) order, permutation, coordinates and pull table of
 * the fluid cells of w's flag grid, ranked by flag_rank; the node arrays
 * perm and coord start at the domain's first node, nbr at the table's, whose
 * node word_base is the domain's first.  Enqueued on st; the Morton order
 * waits for it. */
int flag_tables(const GeomWork &w, int nx, int ny, int nz, int num_p, int ordering,
                int remote_wins, int halfway, int n, long long npad, int *perm, uint16_t *coord,
                uint32_t *nbr, long long rows, uint32_t word_base, uint32_t rest_word,
                cudaStream_t st)
{
    const size_t cells = (size_t)nx * ny * nz;
    TableArgs a;
    a.lexbits = w.lexbits;
    a.lexoffs = w.lexoffs;
    a.obits = a.ooffs = nullptr;
    a.g = Grid{nx, ny, nz, ceil_log2i(nx), ceil_log2i(ny), ceil_log2i(nz),
               ordering == PLB_ORDER_MORTON};
    a.slab = nz / num_p;
    a.remote_wins = remote_wins;
    a.halfway = halfway;
    a.n = n;
    a.npad = npad;
    a.rows = rows;
    a.word_base = word_base;
    a.rest_word = rest_word;
    a.perm = perm;
    a.coord = coord;
    a.nbr = nbr;
    int rc = PLB_OK;
    char *block = nullptr;
    const int bits = a.g.morton ? a.g.bx + a.g.by + a.g.bz : 0;
    if (bits > 40) return PLB_ERR_ARG;
    if (n == 0) return PLB_OK;
    if (!a.g.morton) {
        k_assign_from_flag<true><<<gsz(cells, 256), 256, 0, st>>>(a, cells);
        CKG(cudaGetLastError());
        k_nbr_from_flag<true><<<gsz((size_t)n, 128), 128, 0, st>>>(a);
        CKG(cudaGetLastError());
        return PLB_OK;
    }
    {
        const size_t owords = (((size_t)1 << bits) + 31) / 32;
        const size_t lines = up256(owords * 4);
        CKG(plb_cuda_malloc(&block, 3 * lines + up256(scan_tmp_bytes(owords))));
        uint32_t *obits = (uint32_t *)block, *ooffs = (uint32_t *)(block + lines),
                 *ocnt = (uint32_t *)(block + 2 * lines);
        CKG(cudaMemsetAsync(obits, 0, owords * 4, st));
        k_mark_order<<<gsz(cells, 256), 256, 0, st>>>(w.lexbits, a.g, cells, obits);
        CKG(cudaGetLastError());
        k_popc_words<<<gsz(owords, 256), 256, 0, st>>>(obits, ocnt, owords);
        CKG(cudaGetLastError());
        rc = scan_words(ocnt, ooffs, owords, (uint32_t *)(block + 3 * lines), st);
        if (rc != PLB_OK) goto done;
        a.obits = obits;
        a.ooffs = ooffs;
        k_assign_from_flag<false><<<gsz(cells, 256), 256, 0, st>>>(a, cells);
        CKG(cudaGetLastError());
        k_nbr_from_flag<false><<<gsz((size_t)n, 128), 128, 0, st>>>(a);
        CKG(cudaGetLastError());
    }
done:
    if (block) {
        cudaStreamSynchronize(st);
        cudaFree(block);
    }
    return rc;
}

}  // namespace plb
