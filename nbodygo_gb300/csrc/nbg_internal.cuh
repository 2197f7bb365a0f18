/*
 * nbg_internal.cuh - device-side layout of a context and the kernel entry
 * points shared between the translation units of libnbgpu.so.
 *
 * HBM layout (one context, capacity C bodies):
 *   BodyArrays: 20 FP64 arrays, 2 int64 arrays and 1 u32 flag array of C
 *   elements each (structure of arrays, 180 B per body).  A second BodyArrays
 *   set of the same size receives the compacted collection in Cycle and is
 *   copied back.  Flags hold NBG_F_* in bits 0..7 and the collision
 *   behaviour in bits 8..9.
 *   Mixed form only: jhi/jlo float4 per body (x_hi, y_hi, z_hi, m/m_scale)
 *   and (x_lo, y_lo, z_lo, radius) = 32 B per body, rebuilt every cycle; one
 *   float4 origin per 512-body i-tile; S x 3 x C FP64 partial sums.
 *   Events: one u64 key per detected (i, j) pair: i << 32 | j << 2 | type.
 */
#ifndef NBG_INTERNAL_CUH
#define NBG_INTERNAL_CUH

#include <cstddef>
#include <cstdint>
#include <cuda_runtime.h>

#include "../../include/nbgpu.h"

typedef long long ll;
typedef unsigned long long ull;

#define NBG_BEHAVIOR_SHIFT 8
#define NBG_BEHAVIOR(flags) (((flags) >> NBG_BEHAVIOR_SHIFT) & 3u)
#define NBG_LIVE_MASK (NBG_F_EXISTS | NBG_F_FRAGMENTING)

/* event key type field */
#define NBG_EVT_COLL_IJ 0u /* collision(i, j)      */
#define NBG_EVT_SUB_IJ 1u  /* subsume(i absorbs j) */
#define NBG_EVT_SUB_JI 2u  /* subsume(j absorbs i) */

#define NBG_MAX_BODIES ((ll)1 << 30) /* event keys pack i and j in 30 bits */
#define NBG_MAX_SIMS 2048            /* Hilbert keys of several sims carry the sim in 11 bits */

#define NBG_NF64 20
struct BodyArrays {
    /* the FP64 fields, in this order, are f64[0..19] */
    double *x, *y, *z, *vx, *vy, *vz, *m, *rad, *fx, *fy, *fz, *ff, *fs, *rest;
    double *fr_rad, *fr_newrad, *fr_mass, *fr_cx, *fr_cy, *fr_cz;
    ll *fr_cnt, *id;
    unsigned *flags;
};

/* Control block in device memory; kernels of a cycle read and update it, so
 * a captured graph of one cycle can be replayed. */
struct DevCtl {
    ll n;            /* bodies in the array */
    ll next_id;      /* NextId counter */
    ull cycle;       /* cycle index (fragment generator key) */
    ull seed;
    double dt, R;
    int error;       /* sticky NBG_E_* raised by a kernel */
    int pad0;
    ll error_need;   /* for NBG_E_OVERFLOW: the size that would have fitted */
    int error_what;  /* 1 = bodies, 2 = events, 3 = fragments, 4 = partials, 5 = octree nodes,
                      * 6 = symmetric kernel j-partial units, 7 = inconsistent event links,
                      * 8 = a bulk copy into shared memory that did not complete */
    int splits;      /* mixed: chunks the pair work is cut into (C) */
    ll work_total;   /* mixed: pair work W in (i-tile, j-body) units */
    /* per-cycle values */
    ll ev_count;     /* detected events (may exceed capacity) */
    ll frag_total;   /* fragments emitted this cycle */
    ll n_keep;       /* bodies that survive Cycle */
    ll n_host_adds;  /* adds staged by the host for this cycle */
    ll n_before;     /* bodies at the start of the cycle */
    /* mixed-form reductions (float bits as unsigned for atomicMax) */
    unsigned rmax_bits, xmax_bits;
    double m_scale;
    /* mixed form: pairs closer than near_kappa * (extent of the i-tile around
     * its origin) are evaluated in FP64 (set by the host) */
    float near_kappa;
    /* test hook (NBG_OPT_TEST_WAIT_STALL): bytes the bulk-copy shapes add to
     * each mbarrier's expected count, so that no phase completes; 0 */
    unsigned test_tx_extra;
    /* accumulated over the cycles of one nbg_step call */
    ll acc_steps, acc_interactions, acc_events, acc_frags, acc_removed, acc_nan, acc_bh_terms;
    ll rend_n;       /* renderables written by the last cycle */
    ll last_ev_n;    /* resolved events recorded by the last cycle */
    ll cycle_interactions; /* sum over sims of n_s (n_s - 1) at the cycle start */
    ll acc_ev_max;   /* most events one cycle of this nbg_step call detected */
    ll work_next;    /* mixed: next chunk for the persistent CTAs */
    /* Barnes-Hut (k_bh.cu): bounds of the tree bodies as order-preserving
     * integer images of doubles, the tree body count, nodes built, and the
     * largest radius of any body (for the collision query) */
    ull bh_lo[3], bh_hi[3];
    ll bh_count;
    ll bh_nodes;
    ull bh_rmax;
    unsigned bh_next; /* the walk's next 32-body group (one per warp) */
    unsigned bh_slots; /* the walk's child slots handed out */
    unsigned ticket;   /* blocks of the running kernel that have arrived (last_block) */
    unsigned pad3;
    /* Hilbert order of the mixed path (perm): valid while no body changed
     * index; re-sorted when invalid or sort_interval cycles after the last
     * sort (0: NBG_SORT_INTERVAL_DEFAULT).  sort_now is this cycle's decision. */
    int sort_valid;
    int sort_now;
    int sort_interval;
    int order_carried; /* this cycle's compaction carried the order along */
    ull sort_cycle;
};

#define NBG_SORT_INTERVAL_DEFAULT 4

/* Whether this cycle sorts.  Bodies move a small fraction of a tile's size
 * per cycle, so an order a few cycles old still gives compact tiles; which i
 * a tile holds never changes a result's correctness, only its FP32 error
 * and the near-pair count.  An order is dropped (sort_valid = 0) whenever a
 * body changes index or the arrays are replaced: compaction, loads, edits,
 * reallocation, and a cycle that failed and is run again. */
__device__ __forceinline__ void nbg_sort_decide(DevCtl *ctl)
{
    const int k = ctl->sort_interval > 0 ? ctl->sort_interval : NBG_SORT_INTERVAL_DEFAULT;
    const bool now = !ctl->sort_valid || ctl->cycle - ctl->sort_cycle >= (ull)k;
    ctl->sort_now = now;
    if (now) {
        ctl->sort_valid = 1;
        ctl->sort_cycle = ctl->cycle;
    }
}

/* events sorted by one block in shared memory; more take the multi-block
 * radix sort (when the cycle's launches include it) */
#define NBG_EV_BLOCK_SORT 4096

/* mixed: pairs closer than this factor x the i-body's distance from its
 * tile origin take the near-pair pass (NBG_OPT_NEAR_PPM changes it) */
#define NBG_NEAR_KAPPA_DEFAULT 0.05f
/* collections of at most this many bodies use twice the near-pair factor */
#define NBG_NEAR_SMALL_N 2048
/* In a collection of at most this many bodies the one-sided kernels leave the
 * heaviest body's pull to k_mix_out, which adds it in FP64.  One body, a star,
 * may carry nearly all of every other's force, and then the FP32 error of that
 * one term is the body's, most of it the rounding of the offset from the tile's
 * origin; in larger collections the tiles are smaller next to the distances.
 * Force error of disks of 500 / 1,000 / 2,000 / 3,000 bodies around a star, the
 * star's own left out (L2, mean of 80): 1.48 / 1.84 / 1.95 / 1.76e-7 with the
 * star in the pair kernel, 1e-14 so (1.28 / 1.35 / 1.54 / 1.55e-7 with tiles of 512
 * along a Z-order curve; from 4,000 bodies on the present tiles are better).  A
 * near-pair factor of 0.25 gives 1.3e-7 and costs 30 to 70% of such a cycle; this,
 * nothing that shows in the cycle of 2,501 Plummer bodies. */
#define NBG_HEAVY_MAX_N 4096
/* seg.heavy: |mass| as FP32 bits, then the complement of the index, so that
 * the largest is the heaviest body, and among equals the first */
__host__ __device__ __forceinline__ ull nbg_heavy_key(unsigned mass_bits, unsigned index)
{
    return mass_bits ? (ull)mass_bits << 32 | (unsigned)~index : 0ull;
}
__host__ __device__ __forceinline__ unsigned nbg_heavy_index(ull key) { return ~(unsigned)key; }

/* A collection may hold several independent simulations stored one after
 * another: sim s occupies bodies [off[s], off[s+1]) and bodies of different
 * sims never interact.  Events, fragments and adds stay inside their sim, so
 * each sim follows the reference's cycle exactly as if it were alone. */
struct SimSegs {
    int nsims;
    ll *off;         /* [nsims+1] */
    ll *tile_off;    /* [nsims+1] plain kernel: 64-body i-tiles before sim s */
    ll *mtile_off;   /* [nsims+1] mixed kernel: 512-body i-tiles before sim s */
    ll *item_off;    /* [nsims+1] mixed kernel: pair work before sim s, in (i-tile, j-body)
                      * units: sim s holds (its i-tiles) x n_s of them */
    ll *keep;        /* [nsims]   bodies of sim s that survive Cycle */
    ll *frag;        /* [nsims]   fragments sim s emits this cycle */
    ll *frag_start;  /* [nsims+1] */
    ll *hadd;        /* [nsims]   host adds staged for sim s */
    ll *hadd_start;  /* [nsims+1] */
    ll *keep_start;  /* [nsims+1] */
    ll *new_off;     /* [nsims+1] layout after Cycle */
    unsigned *xmax_bits; /* [nsims] mixed: |x| max of sim s (Hilbert grid) */
    ull *heavy;          /* [nsims] mixed: sim s's heaviest body (NBG_HEAVY_MAX_N), 0 = none */
};

/* bytes of the SimSegs arrays for nsims sims (one allocation, carved by
 * nbg_seg_carve: 12 64-bit arrays and 2 32-bit arrays of nsims + 1) */
#define NBG_SEG_BYTES(ns) ((size_t)((ns) + 1) * 8 * 12 + (size_t)((ns) + 1) * 4 * 2 + 256)

static inline SimSegs nbg_seg_carve(void *base, int nsims)
{
    SimSegs s;
    const size_t m = (size_t)nsims + 1;
    ll *p = (ll *)base;
    s.nsims = nsims;
    s.off = p;
    s.tile_off = p + m;
    s.mtile_off = p + 2 * m;
    s.item_off = p + 3 * m;
    s.keep = p + 4 * m;
    s.frag = p + 5 * m;
    s.frag_start = p + 6 * m;
    s.hadd = p + 7 * m;
    s.hadd_start = p + 8 * m;
    s.keep_start = p + 9 * m;
    s.new_off = p + 10 * m;
    s.heavy = (ull *)(p + 11 * m);
    s.xmax_bits = (unsigned *)(p + 12 * m) + m; /* the first 32-bit array is spare */
    return s;
}

/* sim holding position k of a segmented array: the largest s with
 * off[s] <= k (empty sims are skipped) */
__device__ __forceinline__ int nbg_sim_of(const ll *off, int nsims, ll k)
{
    int lo = 0, hi = nsims - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (off[mid] <= k)
            lo = mid;
        else
            hi = mid - 1;
    }
    return lo;
}

/* Barnes-Hut octree of one collection, nodes in depth-first order */
struct BhTree {
    ull *key[2];        /* octant-path keys (radix ping-pong) */
    unsigned *val[2];   /* body index (ping-pong partner) */
    unsigned *hist;     /* radix digit histogram */
    unsigned *digits;   /* and each pass's digit totals */
    ll *base;           /* nodes starting at each sorted position, then their scan */
    ll *blk;            /* per-block sums of that scan */
    double *mass, *mx, *my, *mz, *cx, *cy, *cz, *half;
    float4 *fa, *fb;    /* mixed walk, by slot: (cm hi xyz, mass / root mass), (cm lo xyz, opening r^2);
                         * FP64 walk: (cm hi xyz, opening r^2), (cm lo xyz, 0) */
    double2 *rec;       /* FP64 walk, by slot: (cm x, y), (cm z, mass) */
    double *shalf;      /* and half size */
    int4 *fc;           /* by slot: (first child's slot, children | flags << 8, start, end) */
    float4 *fd;         /* collision query: the node's cube (centre xyz, half) in FP32 */
    int *skip, *start, *end, *first;
    int *cbase;            /* slot of the first of the node's children */
    unsigned char *ccount; /* and how many there are */
    int *slot;             /* the node's own slot */
    int *parent;           /* the node's parent, -1 for a root */
    unsigned char *flags;
    /* one tree per collection, all in one depth-first node array: per
     * collection s its bounding box (sbox[6 s ..]: lo xyz, hi xyz as
     * order-preserving integers), tree bodies (scount), first sorted
     * position (stree, [nsims + 1]), root node (sroot, [nsims + 1]: the nodes
     * of s are [sroot[s], sroot[s + 1])), first 32-body walk group (sgrp,
     * [nsims + 1]) and first unit of the mixed walk (sunit, [nsims + 1]) */
    ull *sbox;
    ll *scount, *stree, *sroot, *sgrp, *sunit;
    ll node_cap;
};

struct CycleBufs {
    SimSegs seg;
    BodyArrays a;       /* the collection */
    BodyArrays b;       /* compaction target */
    BodyArrays adds;    /* host adds staged for the next Cycle (arrival order) */
    BodyArrays frags;   /* fragments emitted this cycle (arrival order) */
    ll cap, frag_cap, adds_cap;
    ull *ev_keys;
    ull *ev_sort;       /* ping-pong partner of ev_keys for the multi-block event sort */
    ll *ev_hist;        /* its digit histogram and chunk sums (nbg_sort_scratch_hist(ev_cap)) */
    ll ev_cap;
    int ev_radix;       /* this cycle's launches include the multi-block event sort and the
                         * resolution's links (dataflow order) */
    /* resolution links, for cycles beyond the one-block sort: incidence keys
     * (ping-pong, 2 ev_cap each) and their histogram; per event (processing
     * index) the next event on each of its bodies, the count of unresolved
     * predecessors, and the frontier lists (2 ev_cap); each sim's event range */
    ull *inc[2];
    ll *inc_hist;
    ll *ev_link;
    int *ev_pend;
    ll *ev_front;
    ll *ev_lo;
    nbg_event *ev_out;  /* resolved events of the last cycle */
    nbg_renderable *rend;
    ll *blk_sum;        /* per-block counts for the scans */
    ll *blk_off;
    ll nblk_cap;
    /* mixed form (indexed by sorted position) */
    float4 *jhi, *jlo;
    float4 *tile_c;     /* per i-tile: origin (xyz) and a radius holding its bodies (w) */
    float2 *tile_r;     /* per i-tile: its bodies' largest re-centred coordinate and radius (NULL: not kept) */
    int2 *tile_rng;     /* per i-tile: the first and last chunk that share it (NULL: not kept) */
    float4 *iprep;      /* per sorted position: re-centred x, y, z and near-pair threshold */
    double *part;
    unsigned *perm;     /* sorted position -> body index */
    unsigned *skey[2];  /* radix-sort keys (ping-pong) */
    unsigned *sval;     /* radix-sort values (ping-pong partner of perm) */
    unsigned *shist;    /* the spatial order's digit totals and histogram (nbg_order_scratch) */
    ll part_doubles;    /* size of part */
    int work_cap;       /* most CTAs the mixed pair work is divided among (0 = slots) */
    int slots;          /* resident CTAs of the mixed kernel on this device */
    int mix_variant;    /* shape of the mixed pair kernel (see nbg_mix_variant_info) */
    float *jpart;       /* symmetric kernel: FP32 j sums per unit, 3 x itile each */
    ll jpart_units;     /* units jpart holds */
    int itile;          /* i-bodies per work item of that shape */
    /* render ring in mapped host memory (device addresses; NULL: none) */
    nbg_ring_slot *ring_head;
    nbg_renderable *ring_rend;
    ll ring_cap;
    int ring_slots;
    int bh;             /* forces from the Barnes-Hut octree */
    int bh_shape;       /* register cap of the mixed walk: 0, 1, 2 = 4, 5, 6 CTAs per SM */
    int sms;            /* streaming multiprocessors of the device */
    BhTree t;
};

/* Grid of a grid-stride kernel over `items` items, 256 threads per CTA:
 * one CTA per 256 items, at most `per_sm` CTAs per streaming multiprocessor
 * of the device the buffers live on. */
static inline int nbg_flat_grid(const CycleBufs &cb, ll items, int per_sm = 16)
{
    const ll most = (ll)(cb.sms > 0 ? cb.sms : 1) * per_sm;
    ll g = (items + 255) / 256;
    if (g > most) g = most;
    return (int)(g < 1 ? 1 : g);
}

/* Shapes of the mixed pair kernel the autotuner chooses from. */
struct MixVariantInfo {
    int block, k, jt, unroll;
};
#define NBG_MIX_VARIANTS NBG_MIX_SHAPES
/* the symmetric kernel (each unordered pair once, k_pair_sym): shapes 15
 * and 16 (registers capped for 3 and 4 CTAs per SM) */
#define NBG_MIX_SYM 15
__host__ __device__ __forceinline__ bool nbg_mix_is_sym(int variant)
{
    return variant == NBG_MIX_SYM || variant == NBG_MIX_SYM + 1;
}
#define NBG_MIX_MIN_ITILE 256
#define NBG_MIX_MAX_ITILE 512
/* The one-sided pair work is cut into at most NBG_MIX_CHUNKS_PER_CTA chunks
 * per resident CTA, each of at least NBG_MIX_MIN_WORK (i-tile, j-body) units;
 * a collection too small for NBG_MIX_FINE_CHUNKS of those per CTA is cut
 * into that many smaller ones, of at least NBG_MIX_FLOOR_WORK units.  Cycle
 * time of a Plummer sphere on GB300, us, 2,048 units a chunk as before -> now:
 * 2,501 bodies 619 -> 163, 20,011 bodies 1,137 -> 355, 50,001 1,330 -> 1,180;
 * 4 or 16 chunks per CTA in place of 8 are within 5 % of it, and 512 units in
 * place of 1,024 cost 4 % at 50,001 bodies in partial-sum traffic. */
#define NBG_MIX_MIN_WORK 1024
#define NBG_MIX_FINE_CHUNKS 8
#define NBG_MIX_FLOOR_WORK 32
#define NBG_MIX_CHUNKS_PER_CTA 32

/* floor(a b / c) for 0 <= a, 0 < c, without forming a b */
__host__ __device__ __forceinline__ ll nbg_mul_div(ll a, ll b, ll c)
{
    return a * (b / c) + a * (b % c) / c;
}

/* The mixed pair work of a cycle is W units, (i-tile, j-body) pairs in sim,
 * i-tile, j order, cut into C chunks that persistent CTAs take from an
 * atomic counter.  The cut is guided: the first C/4 chunks split the first
 * three quarters of the work evenly and the other chunks the last quarter,
 * so the chunks still running when the counter runs out are a ninth of the
 * first ones and the CTAs finish close together.  The boundaries depend on
 * C and W alone, never on timing.  With W >= 32 C (one-sided; the smallest
 * chunks hold W / (3 C) units) or W >= 4 C (symmetric) every chunk holds
 * work.  This is the first unit of chunk c (c = C gives W). */
__host__ __device__ __forceinline__ ll nbg_chunk_start(ll c, int C, ll W)
{
    const int C1 = C / 4;
    const ll W1 = C1 > 0 ? W - W / 4 : 0;
    if (c <= C1) return C1 > 0 ? nbg_mul_div(c, W1, C1) : 0;
    return W1 + nbg_mul_div(c - C1, W - W1, C - C1);
}

/* the chunk that holds unit u (0 <= u < W) */
__host__ __device__ __forceinline__ int nbg_work_chunk(ll u, int C, ll W)
{
    const int C1 = C / 4;
    const ll W1 = C1 > 0 ? W - W / 4 : 0;
    ll c0, c1;
    if (u < W1) {
        c0 = (ll)((double)u * C1 / (double)W1);
        c0 = c0 < 0 ? 0 : (c0 > C1 - 1 ? C1 - 1 : c0);
        c1 = C1 - 1;
    } else {
        c0 = C1 + (ll)((double)(u - W1) * (C - C1) / (double)(W - W1));
        c0 = c0 < C1 ? C1 : (c0 > C - 1 ? C - 1 : c0);
        c1 = C - 1;
    }
    /* the estimate is off by at most one either way */
    while (c0 > 0 && nbg_chunk_start(c0, C, W) > u) c0--;
    while (c0 < c1 && nbg_chunk_start(c0 + 1, C, W) <= u) c0++;
    return (int)c0;
}

/* Partial sums of the mixed pair kernel: chunk c's share of i-tile g (global
 * tile index) is slot g + c, 3 x itile doubles; no two (tile, chunk) pairs
 * that both hold work share a slot, since chunks are contiguous and ordered.
 * Slots needed: tiles + C - 1, tiles <= cap / itile + sims. */
#define NBG_PART_DOUBLES(cap, chunks, itile) \
    (3 * ((ll)(cap) + (ll)(itile) * ((ll)(chunks) + NBG_MAX_SIMS + 2)))

/* 10 bits spread three apart */
__host__ __device__ __forceinline__ unsigned nbg_spread10(unsigned v)
{
    v &= 0x3ffu;
    v = (v | (v << 16)) & 0x030000ffu;
    v = (v | (v << 8)) & 0x0300f00fu;
    v = (v | (v << 4)) & 0x030c30c3u;
    v = (v | (v << 2)) & 0x09249249u;
    return v;
}

/* Index of cell (x, y, z) of a 2^bits cube along the Hilbert curve (bits <=
 * 10), by Skilling's transpose method (Programming the Hilbert curve, AIP
 * Conf. Proc. 707, 2004): the inverse undo of the rotations from the top bit
 * down, Gray encoding, then the three words' bits interleaved. */
__host__ __device__ __forceinline__ unsigned nbg_hilbert(unsigned x, unsigned y, unsigned z, int bits)
{
    unsigned X[3] = {x, y, z};
    for (unsigned q = 1u << (bits - 1); q > 1u; q >>= 1) {
        const unsigned p = q - 1u;
        for (int i = 0; i < 3; i++) {
            if (X[i] & q) {
                X[0] ^= p;
            } else {
                const unsigned t = (X[0] ^ X[i]) & p;
                X[0] ^= t;
                X[i] ^= t;
            }
        }
    }
    X[1] ^= X[0];
    X[2] ^= X[1];
    unsigned t = 0;
    for (unsigned q = 1u << (bits - 1); q > 1u; q >>= 1)
        if (X[2] & q) t ^= q - 1u;
    return (nbg_spread10(X[0] ^ t) << 2) | (nbg_spread10(X[1] ^ t) << 1) | nbg_spread10(X[2] ^ t);
}

#define NBG_SCAN_BLOCK 1024
#define NBG_SCAN_ITEMS 4
#define NBG_SCAN_TILE (NBG_SCAN_BLOCK * NBG_SCAN_ITEMS)

#define NBG_MIX_BLOCK 128
#define NBG_MIX_K 4
#define NBG_MIX_ITILE (NBG_MIX_BLOCK * NBG_MIX_K)

/* The shape of a context that was not given one.
 *
 * One-sided, 256 bodies a tile: with j tiles of 128 bodies (shape 6: shorter
 * careful passes) for collections below NBG_MIX_FEW_N, of 256 (shape 2: 5%
 * faster once near pairs are few) otherwise.  Shapes 0 / 2 / 6, pair pass in us:
 * Plummer 2,000 bodies 110 / 97 / 97, 20,000 424 / 227 / 202, 50,000 1,053 /
 * 1,009 / 1,012, 131,072 6,652 / 6,351 / 6,675; shapes 2 / 6, 512 spheres of 2,048
 * 3,886 / 3,049, 128 of 8,192 3,928 / 3,760, 48 of 16,384 5,127 / 5,208.
 *
 * The symmetric kernel when every collection has NBG_MIX_SYM_MIN_N bodies (in
 * smaller ones most block pairs hold near pairs: 128 Plummer spheres of 8,192
 * take 6,168 us for 3,928 one-sided, 40 of 20,000 6,846 for 6,276, 30 of 24,000
 * 6,160 for 6,676, 4 of 50,000 3,249 for 3,819; 200 of 256 to 32,768 8,843 for
 * 8,311.  A batch of balls, spheres and disks gains: 512 of 256 to 32,768 20.2 ms
 * for 22.4, at a force error of 1.84e-7 for 1.49e-7, the worst body's 2.6e-6 of its
 * term scale for 2.1e-6; that is left to the autotuner) and there
 * are NBG_MIX_SYM_MIN_UNITS block pairs in all, as one collection of 98,304 makes
 * (fewer share unevenly, and those around a large body take longest).
 * One-sided against symmetric, in ms, for a uniform ball / a disk around a
 * star: 1.65 / 1.84 and 1.54 / 2.29 at 65,536 bodies, 3.61 / 3.74 and 2.84 /
 * 3.85 at 98,304, 6.34 / 6.45 and 4.91 / 5.68 at 131,072, 99.9 / 86.4 and
 * 75.4 / 66.1 at 524,288.  Its j partials grow with the square of the body
 * count (6 KB a block pair); more than an eighth of the device's memory is not
 * taken unasked. */
#define NBG_MIX_ONE_SIDED 2
#define NBG_MIX_ONE_SIDED_FEW 6
#define NBG_MIX_FEW_N 32768
#define NBG_MIX_SYM_MIN_N 24576
#define NBG_MIX_SYM_MIN_UNITS 18528
static inline int nbg_default_shape(int nsims, const ll *counts, unsigned long long device_bytes)
{
    unsigned long long units = 0;
    ll least = 0, most = 0;
    for (int s = 0; s < nsims; s++) {
        least = s == 0 || counts[s] < least ? counts[s] : least;
        most = counts[s] > most ? counts[s] : most;
        const unsigned long long T = ((unsigned long long)counts[s] + NBG_MIX_ITILE - 1) / NBG_MIX_ITILE;
        units += T * (T + 1) / 2;
    }
    const unsigned long long unit_bytes = 3ull * NBG_MIX_ITILE * sizeof(float);
    if (least >= NBG_MIX_SYM_MIN_N && units >= NBG_MIX_SYM_MIN_UNITS &&
        units + units / 4 <= device_bytes / 8 / unit_bytes)
        return NBG_MIX_SYM;
    return most < NBG_MIX_FEW_N ? NBG_MIX_ONE_SIDED_FEW : NBG_MIX_ONE_SIDED;
}
#define NBG_MIX_JT 256

/* The reference's event rules (body.go:174-184): the event type for bodies
 * i, j with behaviours bi, bj, radii ri, rj at distance dist, or -1. */
__device__ static inline int nbg_detect_event(unsigned bi, unsigned bj, double ri, double rj, double dist)
{
    const bool ei = (bi == NBG_ELASTIC || bi == NBG_FRAGMENT);
    const bool ej = (bj == NBG_ELASTIC || bj == NBG_FRAGMENT);
    if (ei && ej) return (int)NBG_EVT_COLL_IJ;
    if (bi == NBG_SUBSUME || bj == NBG_SUBSUME) {
        if (ri > rj && dist <= ri) return (int)NBG_EVT_SUB_IJ;
        if (rj > ri && dist <= rj) return (int)NBG_EVT_SUB_JI;
    }
    return -1;
}

/* appends event (i, j, type) to the list (the count may pass the capacity:
 * the host grows the list and re-runs the cycle) */
__device__ static inline void nbg_emit_event(DevCtl *ctl, ull *keys, ll cap, ll i, ll j, int type)
{
    const ll slot = (ll)atomicAdd((unsigned long long *)&ctl->ev_count, 1ull);
    if (slot < cap) keys[slot] = ((ull)i << 32) | ((ull)j << 2) | (ull)type;
}

/* k_bh.cu (compiled with --fmad=false) */
int nbg_bh_alloc(BhTree &t, ll cap, ll node_cap);
void nbg_bh_free(BhTree &t);
void nbg_launch_bh(const CycleBufs &cb, DevCtl *ctl, cudaStream_t st, bool mixed);
int nbg_bh_launches(const CycleBufs &cb, bool mixed); /* kernels nbg_launch_bh launches */

/* k_cycle.cu (compiled with --fmad=false) */
void nbg_launch_begin(const CycleBufs &cb, DevCtl *ctl, cudaStream_t st, bool direct);
/* the start of a whole cycle: begin, and the fragments it emits */
void nbg_launch_begin_cycle(const CycleBufs &cb, DevCtl *ctl, cudaStream_t st, bool direct);
int nbg_cycle_launches(const CycleBufs &cb, bool carry_order);
void nbg_launch_pair_fp64(const CycleBufs &cb, DevCtl *ctl, cudaStream_t st);
void nbg_launch_after_pair(const CycleBufs &cb, DevCtl *ctl, cudaStream_t st, bool carry_order);
/* sim < 0: every collection (the whole array) */
void nbg_launch_remove(const CycleBufs &cb, DevCtl *ctl, int sim, ll count, ll *removed_dev, cudaStream_t st);
void nbg_launch_edits(const CycleBufs &cb, DevCtl *ctl, int sim, const nbg_edit *edits_dev, ll k, int *results_dev,
                      cudaStream_t st);
void nbg_launch_energy(const CycleBufs &cb, DevCtl *ctl, double *out_dev, cudaStream_t st);
void nbg_launch_find(const CycleBufs &cb, DevCtl *ctl, int sim, ll id, ll *idx_dev, cudaStream_t st);
/* dst[k] = src[index[k]], k < n, every field (index on the device) */
void nbg_launch_gather(const CycleBufs &cb, const BodyArrays &src, const BodyArrays &dst, const ll *index_dev, ll n,
                       cudaStream_t st);

/* k_mixed.cu */
void nbg_launch_mixed_prep(const CycleBufs &cb, DevCtl *ctl, cudaStream_t st);
void nbg_launch_mixed_pair(const CycleBufs &cb, DevCtl *ctl, cudaStream_t st);
void nbg_launch_mixed_out(const CycleBufs &cb, DevCtl *ctl, cudaStream_t st);
int nbg_mixed_launches(const CycleBufs &cb); /* kernels of a mixed force pass, after begin */
int nbg_mixed_slots(int device, int variant);
ll nbg_sym_units(ll blocks);
MixVariantInfo nbg_mix_variant_info(int variant);

/* k_sort.cu */
void nbg_launch_spatial_sort(const CycleBufs &cb, DevCtl *ctl, cudaStream_t st);
int nbg_spatial_sort_launches(const CycleBufs &cb);
void nbg_launch_event_radix(const CycleBufs &cb, DevCtl *ctl, cudaStream_t st);
ull *nbg_launch_incidence_radix(const CycleBufs &cb, DevCtl *ctl, int bits, cudaStream_t st);
int nbg_event_radix_launches(const CycleBufs &cb);
ll nbg_sort_scratch_hist(ll cap);
ll nbg_order_scratch(ll cap);

/* k_probe.cu */
int nbg_run_probes(int device, double *fp32, double *fp64, double *mhz);

#endif
