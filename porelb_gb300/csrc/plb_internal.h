/*
 * plb_internal.h - shared definitions of the CUDA translation units.
 */
#ifndef PLB_INTERNAL_H_
#define PLB_INTERNAL_H_

#include <cuda_runtime.h>
#include <stdint.h>

#include "porelb_gpu.h"
#include "plb_ex.h"
#include "plb_fx.h"

/* Every device allocation of the library goes through here, so that a test
 * can make one of them fail on the host (plb_fault_inject_alloc) and drive
 * the out-of-memory paths without touching the GPU. */
cudaError_t plb_dev_malloc(void **p, size_t bytes);
template <typename P>
static inline cudaError_t plb_cuda_malloc(P **p, size_t bytes)
{
    return plb_dev_malloc((void **)p, bytes);
}

namespace plb {

constexpr int Q = 19;

/* D3Q19 set in the reference order (porelb.h:10-50) as constexpr functions:
 * inside fully unrolled loops they fold to immediates. */
__host__ __device__ constexpr int ex(int j)
{
    return (j == 1 || j == 12 || j == 14 || j == 16 || j == 18) ? 1
         : (j == 2 || j == 11 || j == 13 || j == 15 || j == 17) ? -1 : 0;
}
__host__ __device__ constexpr int ey(int j)
{
    return (j == 3 || j == 7 || j == 10 || j == 15 || j == 18) ? 1
         : (j == 4 || j == 8 || j == 9 || j == 16 || j == 17) ? -1 : 0;
}
__host__ __device__ constexpr int ez(int j)
{
    return (j == 5 || j == 7 || j == 9 || j == 12 || j == 13) ? 1
         : (j == 6 || j == 8 || j == 10 || j == 11 || j == 14) ? -1 : 0;
}
/* re[] (porelb.h:44-50): 1<->2, 3<->4, ... */
__host__ __device__ constexpr int opp(int j)
{
    return j == 0 ? 0 : ((j & 1) ? j + 1 : j - 1);
}
/* weight class: 0 -> 1/3, 1 -> 1/18, 2 -> 1/36 */
__host__ __device__ constexpr int wclass(int j)
{
    return j == 0 ? 0 : (j <= 6 ? 1 : 2);
}

/* A neighbour word is the signed 32-bit offset, counted from the start of
 * plane j of the distribution array, of the value node i pulls for
 * direction j: the source node s (0 <= s < npad) of the pull, or for a
 * bounce-back node i's own value of direction re(j) = j +- 1, which lies at
 * i + (re(j) - j) * npad.  One address computation serves both.  Node index
 * N (the "rest slot") holds the initial value of every direction and is
 * never written: links no push or bounce ever writes read it.  Offsets need
 * 2 * npad < 2^31, hence kMaxNodes. */
constexpr long long kMaxNodes = (1LL << 30) - 512;

__host__ __device__ inline uint32_t bounce_word(int j, long long i, long long npad)
{
    return (uint32_t)(i + (long long)(opp(j) - j) * npad);
}

/* The 18 words of a node lie in five rows, four of four words a node and one
 * of two, so that a thread reads them with four 16-byte loads and one 8-byte
 * load.  Where word j of node i is: in rows of `rows` nodes or, rows 0, with
 * the words of 256 nodes together, which is what short words need (the forms
 * without them lose 0.5-2% by it: FP64 96^3 22.5 against 22.1 us, FP16 7.0
 * against 6.8). */
constexpr int kWordNodes = 256;
constexpr int kWordBlock = 18 * kWordNodes;
__host__ __device__ constexpr long long word_in_rows(int j, long long i, long long rows)
{
    return j <= 16 ? (long long)((j - 1) & ~3) * rows + 4 * i + ((j - 1) & 3)
                   : 16 * rows + 2 * i + (j - 17);
}
__host__ __device__ constexpr long long word_in_block(int j, long long i)
{
    return (i >> 8) * kWordBlock + (j <= 16 ? ((j - 1) >> 2) * 1024 + 4 * (i & 255) + ((j - 1) & 3)
                                            : 4096 + 2 * (i & 255) + (j - 17));
}
__host__ __device__ constexpr long long word_at(int j, long long i, long long rows)
{
    return rows ? word_in_rows(j, i, rows) : word_in_block(j, i);
}

/* Short words.  In row order the sources of direction j lie close to the node
 * itself (dz_planes(j) == 0) or to the node's place in the next or the last
 * z-plane, a distance that is nearly the same for neighbouring nodes.  A block
 * of 256 nodes whose sources all lie within 16 bits of those keeps its words
 * as 16-bit distances instead, in the first half of its place: two rows of
 * eight and one of two.  Two more values mean the node's own reversed value
 * and the rest slot.  Each block has its own two plane distances (what they are counted from),
 * so it makes no difference how much the planes' node counts vary; what does
 * not fit are rows at a periodic wrap in y of planes of more than 32k nodes,
 * and Morton order.  A step of the FP32 form, which streams at the copy rate,
 * reads 36 bytes a node less (256^3: 190 -> 163 us, 36 GLUPS). */
constexpr int kShortBias = 32767; /* a distance d in the plane: d + kShortBias */
/* The distance that a block's words count from for dz_planes(j) == 1 (x) and
 * -1 (y), its smallest; x = kWholeWords for a block whose words are whole. */
constexpr int kWholeWords = -0x7f7f7f80; /* every byte 0x80 */
constexpr uint32_t kShortBounce = 0xfffe;
constexpr uint32_t kShortRest = 0xffff;
__host__ __device__ constexpr int dz_planes(int j) { return -ez(j); }
/* the forms whose steps can read short words (see short_words_pay) */
__host__ __device__ constexpr bool short_form(int precision) { return precision == PLB_FP32; }
/* word_at()'s rows for a form, and the words allocated for npad nodes */
__host__ __device__ constexpr long long word_rows(int precision, long long npad)
{
    return short_form(precision) ? 0 : npad;
}
inline size_t word_count(int precision, long long npad)
{
    if (!short_form(precision)) return 18 * (size_t)npad;
    return (size_t)((npad + kWordNodes - 1) / kWordNodes) * kWordBlock;
}

#if defined(__CUDACC__)
/* store the words w[j - 1] of node i */
__device__ __forceinline__ void store_words(uint32_t *nbr, long long i, long long rows,
                                            const uint32_t (&w)[18])
{
#pragma unroll
    for (int q = 0; q < 4; q++)
        *(uint4 *)(nbr + word_at(4 * q + 1, i, rows)) =
            make_uint4(w[4 * q], w[4 * q + 1], w[4 * q + 2], w[4 * q + 3]);
    *(uint2 *)(nbr + word_at(17, i, rows)) = make_uint2(w[16], w[17]);
}

/* the short words of node i (two to an entry) */
__device__ __forceinline__ void load_short(const uint32_t *nbr, long long i, uint32_t (&q)[9])
{
    const uint32_t *p = nbr + (i >> 8) * kWordBlock;
    const int t = (int)(i & 255);
    const uint4 a = __ldg((const uint4 *)p + t), b = __ldg((const uint4 *)p + 256 + t);
    q[0] = a.x; q[1] = a.y; q[2] = a.z; q[3] = a.w;
    q[4] = b.x; q[5] = b.y; q[6] = b.z; q[7] = b.w;
    q[8] = __ldg(p + 2048 + t);
}

/* the pull word of direction j that node i's short words stand for */
__device__ __forceinline__ int short_word(const uint32_t (&q)[9], int j, int i, long long npad,
                                          int2 base, int rest)
{
    const uint32_t pair = q[(j - 1) >> 1];
    const bool high = !(j & 1);
    const uint32_t w = high ? pair >> 16 : pair & 0xffffu;
    const int from = dz_planes(j) == 0 ? -kShortBias : (dz_planes(j) > 0 ? base.x : base.y);
    int o = (i + from) + (int)w;
    if (high ? pair >= (kShortBounce << 16) : w >= kShortBounce) o = i + (opp(j) - j) * (int)npad;
    if (high ? pair >= (kShortRest << 16) : w >= kShortRest) o = rest;
    return o;
}

/* the pull words w[j - 1] of node i, whichever way its block is kept */
__device__ __forceinline__ void words_of(const uint32_t *nbr, const int2 *shorts, long long i,
                                         long long rows, long long npad, int rest, int (&w)[18])
{
    if (shorts && shorts[i >> 8].x != kWholeWords) {
        uint32_t q[9];
        load_short(nbr, i, q);
        const int2 base = shorts[i >> 8];
#pragma unroll
        for (int j = 1; j <= 18; j++) w[j - 1] = short_word(q, j, (int)i, npad, base, rest);
        return;
    }
#pragma unroll
    for (int q = 0; q < 4; q++) {
        const int4 v = __ldg((const int4 *)(nbr + word_at(4 * q + 1, i, rows)));
        w[4 * q] = v.x; w[4 * q + 1] = v.y; w[4 * q + 2] = v.z; w[4 * q + 3] = v.w;
    }
    const int2 v = __ldg((const int2 *)(nbr + word_at(17, i, rows)));
    w[16] = v.x; w[17] = v.y;
}
#endif

/* Per-solve collision coefficients (host-computed from tau and F). */
struct Coeffs {
    /* FP64, in the reference's operation order */
    double omega, om1, k3, force, half_force;
    /* FP32 forms (rounded from the FP64 values) */
    float omega_f, om1_f, c_f, half_force_f;
    float scale, inv_scale; /* deviation storage scale */
    fx::Consts fxk;         /* fixed-point form */
    ex_::Consts exk;        /* bit-exact form */
    int it;                 /* iteration number (the it > 0 rule) */
    /* bit-exact form: a run constant outside the range of the integer
     * multiply's node check (every node then takes the native multiply) */
    int exact_native;
};

struct StepArgs {
    const void *fin;
    void *fout;
    const uint32_t *nbr;  /* word_at() */
    const int2 *shorts;   /* by block of 256 nodes (see kWholeWords); may be NULL */
    const int *perm;      /* new -> reference index (density guard report) */
    long long npad;
    int n;
    Coeffs co;
    /* macros (rho, ux, uy, uz; stride npad) and per-block sums, or NULL */
    double *macro;
    double *partial;  /* [2][gridDim.x]: sum ux, sum rho */
    unsigned long long *err; /* min over (it << 32 | reference index) */
    unsigned int *flags;     /* bit 0: FP16 scale overflow, bit 1: fallback */
    int pf_blocks;           /* L2 prefetch distance in blocks (0 = none) */
    int words_first;         /* the FP64 form's kernels, built for both, load
                                the words before the wait */
    int trigger;             /* Trigger */
};

/* How a step kernel reads its words: whole ones after the wait for the step
 * before, or before it (see words_first_waves); short ones (before it). */
enum WordMode { kWordsLate, kWordsFirst, kWordsShort };

/* Where a step lets the next one's CTAs start (they then wait for this step to
 * complete): see step_trigger. */
enum Trigger { kTriggerStart, kTriggerWaited, kTriggerGathered, kTriggerExit };

/* Waves of resident CTAs up to which a step loads its words before it waits
 * for the step before; above it, the gathers go out as their words arrive.
 * In a short launch most CTAs start while the step before still drains, and
 * their word loads then cost nothing.  In a long one few do, and 18 words
 * held before the first gather cost registers and make the loads burstier
 * (FP32, words first / after: 3.2 / 3.4 us at 92k nodes, 7.0 / 6.7 at 310k;
 * FP16 2.75 / 3.3, 41.2 / 38.6 at 1.4M; fixed-point FP64 24.2 / 24.8 at 310k,
 * 48.0 / 47.1 at 734k, 9 waves). */
constexpr int words_first_waves(int precision)
{
    return precision == PLB_FP64 ? 6
         : precision == PLB_FP64_EXACT || precision == PLB_FP64_FMA ? 20 : 1;
}

/* One sample of a batch (device copy). */
struct SampleDev {
    Coeffs co;
    long long base; /* first node of the sample in the pool */
    int n;          /* fluid nodes */
    int start;      /* batch step at which the sample started */
};

struct BatchArgs {
    const void *fin;
    void *fout;
    const uint32_t *nbr;
    const int2 *shorts;        /* by pool block (see kWholeWords); may be NULL */
    int rest;                  /* the rest slot */
    long long npad;
    const int *blk_list;       /* pool blocks this launch covers (one CTA each,
                                  two for 128-thread CTAs) */
    const int *blk_sample;     /* per 256-node pool block: sample << 9 | nodes of
                                  the sample in the block, -1 = free */
    long long part_stride;     /* pool blocks: stride of the partial-sum rows */
    const SampleDev *samples;
    const int *t_base;         /* batch step counter (device) */
    int t_off;                 /* this launch's step = *t_base + t_off */
    double *macro;             /* may be NULL */
    double *partial;           /* [3][part_stride] by pool block: sum ux, sum rho,
                                  max |stored deviation| */
    unsigned int *serr;        /* per-sample error bits */
    int pf_blocks;             /* L2 prefetch distance in CTAs (0 = none) */
    int trigger;               /* Trigger */
    /* L2 groups: when grp is set, the launch steps group *grp_cur only,
     * pool blocks blk_list[grp[2g] .. grp[2g] + grp[2g + 1]) */
    const int *grp;
    const int *grp_cur;
};

/* Make the pages of a host buffer that a device copy is about to write
 * present (plb_sim.cu). */
void host_populate(void *p, size_t bytes);
/* the same for four rows of n doubles (each may be NULL) */
void host_populate_rows(double *const (&row)[4], size_t n);

/* Exclusive scan of m uint32 counts into offs (device memory); tmp:
 * scan_tmp_bytes(m) bytes. */
size_t scan_tmp_bytes(size_t m);
int scan_words(const uint32_t *cnt, uint32_t *offs, size_t m, uint32_t *tmp, cudaStream_t st);

/* Device geometry (plb_geom.cu): the scratch of one build, in one block. */
struct GeomWork {
    char *block;
    uint8_t *flag;               /* the flag grid */
    uint32_t *lexbits, *lexoffs; /* fluid bitmap, rank of each word's first cell */
    uint32_t *cnt, *tmp, *meta;
};
int geom_alloc(GeomWork *w, int nx, int ny, int nz, int num_p);
void geom_free(GeomWork *w);
int sphere_pack_device(uint64_t seed, int nx, int ny, int nz, double rmin,
                       double rmax, double porosity, uint8_t *dflag,
                       int *num_spheres, double *porosity_out, cudaStream_t st);
int flag_rank(const GeomWork &w, int nx, int ny, int nz, int num_p, int *n, int *slab_start,
              cudaStream_t st);
int flag_tables(const GeomWork &w, int nx, int ny, int nz, int num_p, int ordering,
                int remote_wins, int halfway, int n, long long npad, int *perm, uint16_t *coord,
                uint32_t *nbr, long long rows, uint32_t word_base, uint32_t rest_word,
                cudaStream_t st);

/* Short words for the blocks of nodes lo .. lo + n - 1 (lo a multiple of 256)
 * whose sources are near: fills in the blocks' shorts, counts them in *count
 * (device memory, may be NULL) and, with `rewrite`, rewrites their words. */
cudaError_t shorten_words(uint32_t *nbr, int2 *shorts, long long lo, int n, int rest,
                          bool rewrite, int *count, cudaStream_t st);

/* the node order for n nodes (plb_auto_ordering), with short words or without */
int auto_order(long long n, int nz, int elem_bytes, bool shorts, int device);

/* whether `nodes` nodes step faster with short words */
bool short_words_pay(int precision, long long nodes);

/* Launch shape of a handle's steps. */
struct StepLaunch {
    int block;       /* threads per CTA */
    int variant;     /* register budget (plb_params.kernel_variant) */
    int wave;        /* CTAs resident on the device at once (0: not planned) */
    int words;       /* WordMode */
    int trigger;     /* Trigger */
};

/* default threads per CTA of the step on n nodes (current device) */
int step_block(int precision, int n);
/* fill in the rest of the shape for n nodes, given block and variant */
void plan_step(int precision, int n, StepLaunch *l);
/* L2 prefetch distance in CTAs of a plain or pool step launch (0: none) */
int prefetch_ctas(int precision, long long nodes, int wave, bool pool, bool shorts, int want);
/* launch one step of the given precision */
cudaError_t launch_step(int precision, bool macros, const StepArgs &a, const StepLaunch &l,
                        cudaStream_t s);
/* CTAs of `cta` threads of the batch step kernel resident on the device at
 * once (0 if unknown) */
int batch_wave_blocks(int precision, int cta);
/* default threads per CTA of the batch step (128 or 256) */
int batch_default_cta(int precision);

/* The batch step kernel (one BatchArgs argument) of a storage form with
 * CTAs of `cta` threads (128 or 256; pool blocks of 256 nodes, 256 / cta
 * CTAs each) for a launch of `grid` CTAs, for a graph kernel node; NULL for
 * another size. */
constexpr int kBatchBlock = 256;
const void *batch_step_kernel(int precision, bool macros, int cta, int grid, bool shorts);
/* its Trigger */
int batch_step_trigger(int precision, int cta, int grid, bool shorts);

/* Fill the coefficients from tau, F and the storage scale. */
void make_coeffs(double tau, double force, float scale, Coeffs *c);

}  // namespace plb

#endif
