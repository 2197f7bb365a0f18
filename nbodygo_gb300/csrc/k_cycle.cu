/*
 * k_cycle.cu - kernels of one compute cycle except the mixed-precision pair
 * kernel: the plain FP64 pair kernel, fragment emission, event ordering,
 * collision resolution, integration, compaction, and the cycle-boundary
 * edits (RemoveBodies, ModBody, GetBody).
 *
 * This file must be compiled with --fmad=false (and -DNBG_NO_FMAD): every
 * FP64 expression then rounds after each operation exactly like the
 * reference's Go code on amd64, which is what makes the plain path
 * bit-identical to the CPU oracle.
 */
#ifndef NBG_NO_FMAD
#error "k_cycle.cu must be compiled with --fmad=false -DNBG_NO_FMAD"
#endif

#include "nbg_exact.h"
#include "nbg_internal.cuh"
#include "nbg_math.h"
#include "nbg_shared.h"

#define FULL_MASK 0xffffffffu

/* ------------------------------------------------------------------------ */
/* block-wide exclusive scan (blockDim.x == NBG_SCAN_BLOCK)                 */
/* ------------------------------------------------------------------------ */

__device__ static ll block_excl_scan(ll v, ll *total)
{
    __shared__ ll warp_tot[NBG_SCAN_BLOCK / 32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    ll x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        ll y = __shfl_up_sync(FULL_MASK, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) warp_tot[w] = x;
    __syncthreads();
    if (w == 0) {
        ll t = warp_tot[lane];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            ll y = __shfl_up_sync(FULL_MASK, t, o);
            if (lane >= o) t += y;
        }
        warp_tot[lane] = t;
    }
    __syncthreads();
    ll excl = x - v + (w > 0 ? warp_tot[w - 1] : 0);
    *total = warp_tot[NBG_SCAN_BLOCK / 32 - 1];
    __syncthreads();
    return excl;
}

/* Exclusive scan of f(0..ns-1) into out[0..ns-1], out[ns] = total, by one
 * block of NBG_SCAN_BLOCK threads; returns the total to every thread. */
template <typename F>
__device__ static ll block_scan_array(int ns, F f, ll *out)
{
    ll carry = 0;
    for (int s0 = 0; s0 < ns; s0 += NBG_SCAN_BLOCK) {
        const int s = s0 + (int)threadIdx.x;
        const ll v = s < ns ? f(s) : 0;
        ll tot;
        const ll ex = block_excl_scan(v, &tot);
        if (s < ns) out[s] = carry + ex;
        carry += tot;
    }
    if (threadIdx.x == 0) out[ns] = carry;
    __syncthreads();
    return carry;
}

/* ------------------------------------------------------------------------ */
/* cycle start                                                              */
/* ------------------------------------------------------------------------ */

/* Per-cycle resets and the work layout of every sim: 64-body tiles of the
 * plain kernel; i-tiles and the pair work of the mixed kernel, and the chunks
 * it is cut into (C: NBG_MIX_CHUNKS_PER_CTA per resident CTA, or work_cap,
 * fewer for small collections, and few enough that the partial-sum slots fit
 * in part_doubles); the interaction count.  One block. */
__device__ static void begin_cycle(DevCtl *ctl, const SimSegs &seg, int slots, int work_cap, int itile,
                                   ll part_doubles, int sym, ll jpart_units)
{
    const int ns = seg.nsims;
    const ll *off = seg.off;
    for (int s = threadIdx.x; s < ns; s += NBG_SCAN_BLOCK) {
        seg.keep[s] = 0;
        seg.frag[s] = 0;
        seg.xmax_bits[s] = 0;
        seg.heavy[s] = 0;
    }
    block_scan_array(ns, [&](int s) { return (off[s + 1] - off[s] + 63) / 64; }, seg.tile_off);
    const ll mtiles = block_scan_array(
        ns, [&](int s) { return (off[s + 1] - off[s] + itile - 1) / itile; }, seg.mtile_off);
    /* one-sided kernel: (i-tile, j-body) units; symmetric kernel: the
     * (block, block) pairs a <= b of each collection, T (T + 1) / 2 of them */
    const ll W = block_scan_array(
        ns,
        [&](int s) {
            const ll T = seg.mtile_off[s + 1] - seg.mtile_off[s];
            return sym ? T * (T + 1) / 2 : T * (off[s + 1] - off[s]);
        },
        seg.item_off);
    ll P = (ll)slots * NBG_MIX_CHUNKS_PER_CTA;
    if (work_cap > 0 && P > work_cap) P = work_cap;
    /* every chunk must hold work: the smallest guided chunk is W / (3 P) */
    ll most = W / 4;
    if (!sym) {
        /* Chunks of NBG_MIX_MIN_WORK units once there are NBG_MIX_FINE_CHUNKS
         * per resident CTA; below that size the chip would idle (10 chunks
         * for 2,501 bodies, one per CTA at 20,011), so the work is cut that
         * finely, down to NBG_MIX_FLOOR_WORK units a chunk. */
        ll fine = (ll)slots * NBG_MIX_FINE_CHUNKS;
        if (fine > W / NBG_MIX_FLOOR_WORK) fine = W / NBG_MIX_FLOOR_WORK;
        most = W / NBG_MIX_MIN_WORK > fine ? W / NBG_MIX_MIN_WORK : fine;
    }
    if (P > most) P = most;
    const ll part_slots = part_doubles / (3ll * itile);
    if (P > part_slots - mtiles + 1) P = part_slots - mtiles + 1;
    if (P < 1) P = 1;
    const bool part_short = mtiles + P - 1 > part_slots;
    /* interactions: sum of n_s (n_s - 1), reusing the keep_start array */
    const ll inter = block_scan_array(
        ns, [&](int s) { const ll m = off[s + 1] - off[s]; return m * (m > 0 ? m - 1 : 0); }, seg.keep_start);
    if (threadIdx.x == 0) {
        ll n = ctl->n;
        ctl->n_before = n;
        ctl->ev_count = 0;
        ctl->frag_total = 0;
        ctl->n_keep = n;
        ctl->rend_n = 0;
        ctl->last_ev_n = 0;
        ctl->rmax_bits = 0;
        ctl->xmax_bits = 0;
        ctl->m_scale = 0.0;
        ctl->splits = (int)P;
        ctl->work_total = W;
        ctl->work_next = 0;
        for (int c = 0; c < 3; c++) {
            ctl->bh_lo[c] = ~0ull;
            ctl->bh_hi[c] = 0ull;
        }
        ctl->bh_count = 0;
        ctl->bh_nodes = 0;
        ctl->bh_rmax = 0ull;
        ctl->bh_next = 0;
        ctl->bh_slots = 0;
        ctl->cycle_interactions = inter;
        if (part_short) {
            ctl->error = NBG_E_OVERFLOW;
            ctl->error_what = 4;
            ctl->error_need = (mtiles + P - 1) * 3ll * itile;
        } else if (sym && W > jpart_units) {
            ctl->error = NBG_E_OVERFLOW;
            ctl->error_what = 6;
            ctl->error_need = W;
        }
    }
    __syncthreads();
}

__global__ void __launch_bounds__(NBG_SCAN_BLOCK) k_begin(DevCtl *ctl, SimSegs seg, int slots, int work_cap, int itile,
                                                          ll part_doubles, int sym, ll jpart_units)
{
    if (ctl->error) return;
    begin_cycle(ctl, seg, slots, work_cap, itile, part_doubles, sym, jpart_units);
}

/* Fragments body k emits this cycle: Compute calls fragment() for a body that
 * exists and is fragmenting (body.go:148-154); the loop of fragcalc.go:96-111
 * emits min(fragments, 101) when fragments > 0. */
__device__ static ll frag_emit_count(const BodyArrays &A, ll k)
{
    unsigned f = A.flags[k];
    if ((f & NBG_LIVE_MASK) != NBG_LIVE_MASK) return 0;
    ll c = A.fr_cnt[k];
    if (c <= 0) return 0;
    return c < NBG_MAX_FRAGS_PER_CYCLE + 1 ? c : NBG_MAX_FRAGS_PER_CYCLE + 1;
}

/* Adds `v` to counter[sim] once per group of lanes that share `sim` (sim < 0:
 * nothing).  Every lane of the warp must call it. */
__device__ static void warp_add_per_sim(ll *counter, int sim, unsigned v)
{
    const unsigned peers = __match_any_sync(FULL_MASK, sim);
    const unsigned t = __reduce_add_sync(peers, v);
    if (sim >= 0 && (int)(threadIdx.x & 31) == __ffs(peers) - 1 && t != 0)
        atomicAdd((unsigned long long *)&counter[sim], (ull)t);
}

/* Sums over the bodies of scan tile `blk` (NBG_SCAN_TILE of them), one block:
 * fragments emitted, bodies kept. */
__device__ static void frag_blocksum(const BodyArrays &A, const DevCtl *ctl, const SimSegs &seg, ll blk, ll *blk_sum)
{
    const ll n = ctl->n;
    const ll base = blk * NBG_SCAN_TILE;
    if (base >= n) return;
    ll s = 0;
    for (int q = 0; q < NBG_SCAN_ITEMS; q++) {
        ll k = base + (ll)threadIdx.x * NBG_SCAN_ITEMS + q;
        if (k < n) {
            const ll c = frag_emit_count(A, k);
            s += c;
            if (c > 0) atomicAdd((unsigned long long *)&seg.frag[nbg_sim_of(seg.off, seg.nsims, k)], (ull)c);
        }
    }
    ll tot;
    block_excl_scan(s, &tot);
    if (threadIdx.x == 0) blk_sum[blk] = tot;
}

__device__ static void keep_blocksum(const BodyArrays &A, const DevCtl *ctl, const SimSegs &seg, ll blk, ll *blk_sum)
{
    const ll n = ctl->n;
    const ll base = blk * NBG_SCAN_TILE;
    if (base >= n) return;
    ll s = 0;
    for (int q = 0; q < NBG_SCAN_ITEMS; q++) {
        /* consecutive lanes take consecutive bodies so a warp mostly sees one sim */
        const ll k = base + (ll)q * NBG_SCAN_BLOCK + threadIdx.x;
        const bool keep = k < n && (A.flags[k] & NBG_F_EXISTS);
        s += keep ? 1 : 0;
        warp_add_per_sim(seg.keep, keep ? nbg_sim_of(seg.off, seg.nsims, k) : -1, keep ? 1 : 0);
    }
    ll tot;
    block_excl_scan(s, &tot);
    if (threadIdx.x == 0) blk_sum[blk] = tot;
}

/* Single-block exclusive scan of the per-block sums, then the per-sim
 * layout.  mode 0: fragment counts, fragment and host-add starts per sim,
 * capacity checks.  mode 1: surviving bodies, keep starts and the layout
 * after Cycle: sim s gets [kept bodies][its fragments][its host adds].
 * mode 2: the block offsets alone. */
__device__ static void scan_blocks(DevCtl *ctl, const SimSegs &seg, const ll *blk_sum, ll *blk_off, int mode, ll cap,
                                   ll frag_cap)
{
    const ll n = ctl->n;
    const ll nb = (n + NBG_SCAN_TILE - 1) / NBG_SCAN_TILE;
    ll carry = 0;
    for (ll b0 = 0; b0 < nb; b0 += NBG_SCAN_BLOCK) {
        ll b = b0 + threadIdx.x;
        ll v = b < nb ? __ldcg(&blk_sum[b]) : 0; /* other blocks' writes */
        ll tot;
        ll ex = block_excl_scan(v, &tot);
        if (b < nb) blk_off[b] = carry + ex;
        carry += tot;
    }
    const int ns = seg.nsims;
    if (mode == 2) {
        __syncthreads();
        return; /* block offsets only (the carried order) */
    }
    if (mode == 0) {
        block_scan_array(ns, [&](int s) { return __ldcg(&seg.frag[s]); }, seg.frag_start);
        const ll hadds = block_scan_array(ns, [&](int s) { return seg.hadd[s]; }, seg.hadd_start);
        if (threadIdx.x == 0) {
            ctl->frag_total = carry;
            ctl->n_host_adds = hadds;
            ll need = n + carry + hadds;
            if (carry > frag_cap) {
                ctl->error = NBG_E_OVERFLOW;
                ctl->error_what = 3;
                ctl->error_need = carry;
            } else if (need > cap) {
                ctl->error = NBG_E_OVERFLOW;
                ctl->error_what = 1;
                ctl->error_need = need;
            }
        }
    } else {
        block_scan_array(ns, [&](int s) { return __ldcg(&seg.keep[s]); }, seg.keep_start);
        block_scan_array(ns, [&](int s) { return __ldcg(&seg.keep[s]) + seg.frag[s] + seg.hadd[s]; }, seg.new_off);
        if (threadIdx.x == 0) ctl->n_keep = carry;
    }
    __syncthreads();
}

/* True in every thread of the block that arrives last of the grid, with the
 * other blocks' writes visible to it: a block sum's scan needs no launch of
 * its own (3 to 5 us each).  No block waits for another. */
__device__ static bool last_block(DevCtl *ctl)
{
    __shared__ unsigned s_last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
        s_last = atomicAdd(&ctl->ticket, 1u) == gridDim.x - 1 ? 1u : 0u;
        if (s_last) ctl->ticket = 0;
    }
    __syncthreads();
    __threadfence();
    return s_last != 0;
}

__global__ void __launch_bounds__(NBG_SCAN_BLOCK) k_frag_count(BodyArrays A, DevCtl *ctl, SimSegs seg, ll *blk_sum,
                                                               ll *blk_off, ll cap, ll frag_cap)
{
    if (ctl->error) return;
    frag_blocksum(A, ctl, seg, blockIdx.x, blk_sum);
    if (last_block(ctl)) scan_blocks(ctl, seg, blk_sum, blk_off, 0, cap, frag_cap);
}

__global__ void __launch_bounds__(NBG_SCAN_BLOCK) k_keep_count(BodyArrays A, DevCtl *ctl, SimSegs seg, ll *blk_sum,
                                                               ll *blk_off)
{
    if (ctl->error) return;
    keep_blocksum(A, ctl, seg, blockIdx.x, blk_sum);
    if (last_block(ctl)) scan_blocks(ctl, seg, blk_sum, blk_off, 1, 0, 0);
}

/* The cycle's start of a collection of one scan tile's capacity: k_begin and
 * k_frag_count by one block.  Launches of a few microseconds each are most of
 * a small collection's cycle: with 10 launches in place of 45 the mixed cycle of
 * 2,501 bodies takes 103 us in place of 161, with 6 in place of 14 the plain
 * cycle of 1,000 bodies 101 in place of 110. */
__global__ void __launch_bounds__(NBG_SCAN_BLOCK) k_begin_small(BodyArrays A, DevCtl *ctl, SimSegs seg, int slots,
                                                                int work_cap, int itile, ll part_doubles, int sym,
                                                                ll jpart_units, ll *blk_sum, ll *blk_off, ll cap,
                                                                ll frag_cap)
{
    if (ctl->error) return;
    begin_cycle(ctl, seg, slots, work_cap, itile, part_doubles, sym, jpart_units);
    if (ctl->error) return; /* the same in every thread after the barrier */
    frag_blocksum(A, ctl, seg, 0, blk_sum);
    __syncthreads();
    scan_blocks(ctl, seg, blk_sum, blk_off, 0, cap, frag_cap);
}

/* ------------------------------------------------------------------------ */
/* K1: plain FP64 force + collision detection                              */
/* ------------------------------------------------------------------------ */

/* One pair of calcForceFrom and Collided (body.go:192-225) with the ordinary
 * operators, for whatever the straight path does not take: bodies that may
 * touch (their comparison and their event), that are not there, massless or
 * the same one, and the operands nbg_exact.h refuses. */
__device__ __noinline__ static void p64_pair_plain(DevCtl *ctl, ull *ev_keys, ll ev_cap, ll i, ll j, unsigned fi,
                                                   unsigned fj, double dx, double dy, double dz, double gmi, double mj,
                                                   double ri, double rj, double &ex, double &ey, double &ez)
{
    ex = ey = ez = 0.0;
    if ((fi & NBG_LIVE_MASK) != NBG_F_EXISTS || j == i) return;
    const double dist = sqrt(dx * dx + dy * dy + dz * dz);
    const double rr = ri + rj;
    const bool coll_i = (fi & NBG_F_COLLIDED) != 0;
    if (!coll_i && dist <= rr) {
        const int type = nbg_detect_event(NBG_BEHAVIOR(fi), NBG_BEHAVIOR(fj), ri, rj, dist);
        if (type >= 0) nbg_emit_event(ctl, ev_keys, ev_cap, i, j, type);
    }
    if ((fj & NBG_LIVE_MASK) != NBG_F_EXISTS || !(coll_i || dist > rr)) return;
    const double force = gmi * mj / (dist * dist);
    ex = force * dx / dist;
    ey = force * dy / dist;
    ez = force * dz / dist;
}

/* Upper bound on the high word of 2 max(r, 0): dist > r_i + r_j for sure when
 * dist's high word is above both bodies' bounds.  NaN and huge radii get the
 * largest value, and their pairs the exact comparison. */
__device__ __forceinline__ int p64_radius_bound(double r)
{
    const int h = __double2hiint(r);
    if (r != r || h >= 0x7fe00000) return 0x7fffffff;
    return h < 0 ? h : h + 0x100000;
}

/* beside a body's flags: it is not live, or its mass (or G times it) is not
 * in nbg_exact.h's range */
#define P64_ODD 0x10000u
__device__ __forceinline__ unsigned p64_flags(unsigned f, double m)
{
    return (f & 0xffffu) | ((f & NBG_LIVE_MASK) == NBG_F_EXISTS && nbx_mass_ok(nbx_bits(m)) ? 0u : P64_ODD);
}

/* One CTA takes a block of up to 32 bodies i of one collection and walks its
 * j in tiles.  Eight warps compute the pair terms of a tile, up to 1,536
 * (i, j), into shared memory; up to three more warps, a lane for each force
 * component of each body, add the tile before it, each body's terms in j
 * order.  So every expression and every addition is the reference's
 * sequential one (the file is compiled with --fmad=false), while a collection
 * of any size fills the chip: the block is cut so that every resident CTA
 * gets the same number of bodies.
 *
 * Bound by the FP64 pipe and the integer pipes together.  The pipe takes
 * 11.6 operations a pair (differences 3, squared distance 5, sums 3 in three
 * warps of 27 lanes for 16,384 bodies) of 19 cycles per SM each, 220 cycles a
 * warp of pairs; the root, four quotients and four products run beside it on
 * integers (nbg_exact.h), some 650 issue cycles a scheduler, 190 a pair warp
 * and SM.  Leaving more products to the pipe, or none of the squares, measured
 * 1-8 % slower.  16,384 Plummer bodies 28.9 -> 8.4 ms a pass, where the
 * compiler's expansion of the root and the divisions kept the FP64 pipe 90 %
 * busy with 68 operations a pair; terms stay on the chip, where storing them
 * all took 48 bytes of traffic a pair and 3.2 GB at 65,536 bodies.  A body's
 * sum is one chain of n dependent additions of 64 cycles at least: that is
 * what a collection of a thousand bodies waits for (174 -> 75 us).  Tiles of
 * 512 pairs, with a barrier three times as often, measured 11.1 ms. */
#define P64_PROD 256
#define P64_THREADS (P64_PROD + 96)
#define P64_PAIRS (6 * P64_PROD) /* most pairs of a tile */
#define P64_IB 32                /* most bodies of a block */
#define P64_JT 192               /* most j of a tile */
#define P64_MINB 2               /* CTAs per SM */
static_assert(P64_JT <= P64_PROD, "a tile's j are loaded one per producer");
static_assert(P64_PROD % P64_IB == 0 && P64_JT % (P64_PROD / 4) == 0, "tiles of whole rounds");
static_assert(P64_PAIRS <= 2048, "the reciprocal of ib is exact below 2048");
static_assert(P64_THREADS - P64_PROD >= 3 * P64_IB, "an adder for every component of a block");
struct P64Shared {
    double term[2][3][P64_PAIRS];
    double jx[2][P64_JT], jy[2][P64_JT], jz[2][P64_JT], jm[2][P64_JT], jr[2][P64_JT];
    double sx[P64_IB], sy[P64_IB], sz[P64_IB], sg[P64_IB], sr[P64_IB];
    ll blk;
    unsigned jf[2][P64_JT], sf[P64_IB];
    int jb[2][P64_JT], sb[P64_IB];
};
/* MANY: several collections */
template <bool MANY>
__global__ void __launch_bounds__(P64_THREADS, P64_MINB) k_pair_fp64(BodyArrays A, DevCtl *ctl, SimSegs seg, ull *ev_keys,
                                                              ll ev_cap)
{
    extern __shared__ double p64_smem[];
    P64Shared &S = *(P64Shared *)p64_smem;
    auto &term = S.term;
    auto &jx = S.jx, &jy = S.jy, &jz = S.jz, &jm = S.jm, &jr = S.jr;
    auto &jf = S.jf;
    auto &jb = S.jb;
    auto &sx = S.sx, &sy = S.sy, &sz = S.sz, &sg = S.sg, &sr = S.sr;
    auto &sf = S.sf;
    auto &sb = S.sb;
    ll &s_blk = S.blk;
    if (ctl->error) return;
    const int tid = threadIdx.x;
    const bool producer = tid < P64_PROD;
    const int ns = seg.nsims;
    /* bodies of a block.  One collection: even shares of the resident CTAs'
     * waves.  Several: 4 to 32, a divisor of the 64-body tiles the layout
     * counts, small enough for four blocks a CTA. */
    int ib;
    ll blocks;
    if (!MANY) {
        const ll n = ctl->n;
        const ll waves = (n + (ll)P64_IB * gridDim.x - 1) / ((ll)P64_IB * gridDim.x);
        ib = waves > 0 ? (int)((n + waves * gridDim.x - 1) / (waves * gridDim.x)) : 1;
        if (ib < 4) ib = 4;
        blocks = (n + ib - 1) / ib;
    } else {
        const ll tiles = seg.tile_off[ns];
        ib = P64_IB;
        while (ib > 4 && tiles * (64 / ib) < 4ll * gridDim.x) ib >>= 1;
        blocks = tiles * (64 / ib);
    }
    const int jmost = P64_PAIRS / ib < P64_JT ? P64_PAIRS / ib : P64_JT; /* j of a tile, at most */
    const unsigned rib = ((1u << 20) + (unsigned)ib - 1u) / (unsigned)ib; /* p / ib = p rib >> 20 for p < 2048 */
    /* the adders: 3 ib threads in a row, one for each component of each body */
    const int comp = producer ? 3 : (tid - P64_PROD) / ib, lane = tid - P64_PROD - comp * ib;
    const bool adder = comp < 3;
    for (;;) {
        if (tid == 0) s_blk = (ll)atomicAdd((unsigned long long *)&ctl->work_next, 1ull);
        __syncthreads();
        const ll B = s_blk;
        if (B >= blocks) break;
        ll s0, n, ibase;
        if (!MANY) {
            s0 = 0;
            n = ctl->n;
            ibase = B * ib;
        } else {
            const int per = 64 / ib;
            const ll T = B / per;
            const int sim = nbg_sim_of(seg.tile_off, ns, T);
            s0 = seg.off[sim];
            n = seg.off[sim + 1];
            ibase = s0 + (T - seg.tile_off[sim]) * 64 + (B - T * per) * ib;
        }
        int jt = jmost;
        if (MANY) {
            if (ibase >= n) { /* past the end of the collection's last 64 bodies */
                __syncthreads(); /* s_blk is rewritten next */
                continue;
            }
            /* Every place of a tile is computed, also past the collection's
             * end, P64_PROD places a round: equal tiles of as few rounds as
             * hold it.  2,048 collections of 8 bodies spent five sixths of the
             * pass past their ends, 318 -> 117 us a cycle, 1,000 of 65 bodies
             * 435 -> 363.  (One collection: a length by block costs 0.6% at
             * 16,384 bodies.) */
            const int unit = P64_PROD / ib, most = jmost / unit;
            const int rounds = ((int)(n - s0) + unit - 1) / unit, tiles = (rounds + most - 1) / most;
            jt = (rounds + tiles - 1) / tiles * unit;
        }
        if (tid < ib) {
            const ll i = ibase + tid;
            const bool valid = i < n;
            sx[tid] = valid ? A.x[i] : 0.0;
            sy[tid] = valid ? A.y[i] : 0.0;
            sz[tid] = valid ? A.z[i] : 0.0;
            sg[tid] = valid ? NBG_G * A.m[i] : 0.0;
            sr[tid] = valid ? A.rad[i] : 0.0;
            sf[tid] = valid ? p64_flags(A.flags[i], sg[tid]) : P64_ODD;
            sb[tid] = valid ? p64_radius_bound(A.rad[i]) : 0;
        }
        auto load_j = [&](ll jbase, int buf) {
            const ll j = jbase + tid;
            if (tid < jt && j >= n) {
                jf[buf][tid] = P64_ODD; /* past the end: neither live nor near */
                jx[buf][tid] = jy[buf][tid] = jz[buf][tid] = jm[buf][tid] = 0.0;
                jr[buf][tid] = __longlong_as_double(0x7ff8000000000000ll);
            } else if (tid < jt) {
                jx[buf][tid] = A.x[j];
                jy[buf][tid] = A.y[j];
                jz[buf][tid] = A.z[j];
                jm[buf][tid] = A.m[j];
                const double r = A.rad[j];
                jr[buf][tid] = r;
                jb[buf][tid] = p64_radius_bound(r);
                jf[buf][tid] = p64_flags(A.flags[j], jm[buf][tid]);
            }
        };
        /* The straight path: no branch, so that a thread's pairs overlap.
         * Returns whether it holds; if not, the term is meaningless. */
        auto core = [&](int ii, int jj, int buf, double &ex, double &ey, double &ez) -> bool {
            const double dx = jx[buf][jj] - sx[ii];
            const double dy = jy[buf][jj] - sy[ii];
            const double dz = jz[buf][jj] - sz[ii];
            const uint64_t bx = nbx_bits(dx), by = nbx_bits(dy), bz = nbx_bits(dz);
            const double s = dx * dx + dy * dy + dz * dz;
            const nbx_root root = nbx_sqrt(nbx_bits(s));
            const nbx_div &r = root.r;
            const int bound = sb[ii] > jb[buf][jj] ? sb[ii] : jb[buf][jj];
            const nbx_num gm = nbx_mul(nbx_unpack(nbx_bits(sg[ii])), nbx_unpack(nbx_bits(jm[buf][jj])));
            const nbx_num f = nbx_quot(gm, nbx_square(root));
            const nbx_num ax = nbx_mul(f, nbx_unpack(bx)), ay = nbx_mul(f, nbx_unpack(by)),
                          az = nbx_mul(f, nbx_unpack(bz));
            ex = nbx_zero(bx) ? 0.0 : nbx_double(nbx_pack(nbx_quot(ax, r)));
            ey = nbx_zero(by) ? 0.0 : nbx_double(nbx_pack(nbx_quot(ay, r)));
            ez = nbx_zero(bz) ? 0.0 : nbx_double(nbx_pack(nbx_quot(az, r)));
            return nbx_diff_ok(bx) && nbx_diff_ok(by) && nbx_diff_ok(bz) && !nbx_zero(bx | by | bz) &&
                   nbx_square_ok(root) && (int)(nbx_div_bits(r) >> 32) > bound;
        };
        auto plain = [&](int ii, int jj, ll jbase, int buf, double &ex, double &ey, double &ez) {
            p64_pair_plain(ctl, ev_keys, ev_cap, ibase + ii, jbase + jj, sf[ii], jf[buf][jj], jx[buf][jj] - sx[ii],
                           jy[buf][jj] - sy[ii], jz[buf][jj] - sz[ii], sg[ii], jm[buf][jj], sr[ii], jr[buf][jj], ex, ey,
                           ez);
        };
        double f = 0.0;
        auto add = [&](ll jbase, int buf) {
            if (adder) {
                const int cnt = n - jbase < jt ? (int)(n - jbase) : jt;
                const double *q = &term[buf][comp][lane];
#pragma unroll 8
                for (int t = 0; t < cnt; t++) f += q[t * ib];
            }
        };
        if (producer) load_j(s0, 0);
        __syncthreads();
        int buf = 0;
        for (ll jbase = s0; jbase < n; jbase += jt, buf ^= 1) {
            if (producer) {
                if (jbase + jt < n) load_j(jbase + jt, buf ^ 1);
                /* pair p of the tile: body p % ib, j p / ib */
                const int np = ib * jt;
#pragma unroll 1
                for (int p = tid; p < np; p += P64_PROD) {
                    const int jj = (int)(((unsigned)p * rib) >> 20), ii = p - jj * ib;
                    double ex, ey, ez;
                    const bool ok = core(ii, jj, buf, ex, ey, ez);
                    if (!ok || ((sf[ii] | jf[buf][jj]) & P64_ODD)) plain(ii, jj, jbase, buf, ex, ey, ez);
                    term[buf][0][p] = ex;
                    term[buf][1][p] = ey;
                    term[buf][2][p] = ez;
                }
            } else if (jbase > s0) {
                add(jbase - jt, buf ^ 1);
            }
            __syncthreads();
        }
        if (!producer && n > s0) {
            const ll last = s0 + (n - s0 - 1) / jt * jt;
            add(last, buf ^ 1);
            const ll i = ibase + lane;
            if (adder && i < n && (sf[lane] & NBG_LIVE_MASK) == NBG_F_EXISTS)
                (comp == 0 ? A.fx : comp == 1 ? A.fy : A.fz)[i] = f;
        }
        __syncthreads(); /* the block's shared data and s_blk are rewritten next */
    }
}

/* ------------------------------------------------------------------------ */
/* K4: order the events (i ascending, then j)                               */
/* ------------------------------------------------------------------------ */

#define SORT_BLOCK 1024
#define SORT_SMEM NBG_EV_BLOCK_SORT

/* Orders the cycle's events by key (i, then j): up to SORT_SMEM in shared
 * memory by one block.  More are left to the multi-block radix sort that
 * follows when radix_follows is set; otherwise this block sorts them in
 * global memory (bitonic, slow but correct). */
__device__ static void sort_events(DevCtl *ctl, ull *keys, ll cap, int radix_follows)
{
    __shared__ ull s[SORT_SMEM];
    __shared__ int bail;
    if (threadIdx.x == 0) {
        bail = ctl->error != 0;
        if (!bail && ctl->ev_count > cap) {
            ctl->error = NBG_E_OVERFLOW;
            ctl->error_what = 2;
            ctl->error_need = ctl->ev_count;
            bail = 1;
        }
        if (!bail && ctl->ev_count > ctl->acc_ev_max) ctl->acc_ev_max = ctl->ev_count;
    }
    __syncthreads();
    if (bail) return;
    const ll cnt = ctl->ev_count;
    if (cnt <= 1 || (cnt > SORT_SMEM && radix_follows)) return;
    ll P = 1;
    while (P < cnt) P <<= 1;
    ull *d = keys;
    if (P <= SORT_SMEM) {
        d = s;
        for (ll k = threadIdx.x; k < P; k += SORT_BLOCK) s[k] = k < cnt ? keys[k] : ~0ull;
    } else {
        for (ll k = cnt + threadIdx.x; k < P; k += SORT_BLOCK) keys[k] = ~0ull;
    }
    __syncthreads();
    for (ll kk = 2; kk <= P; kk <<= 1) {
        for (ll jj = kk >> 1; jj > 0; jj >>= 1) {
            for (ll idx = threadIdx.x; idx < P; idx += SORT_BLOCK) {
                ll ixj = idx ^ jj;
                if (ixj > idx) {
                    bool asc = (idx & kk) == 0;
                    ull a = d[idx], b = d[ixj];
                    if ((a > b) == asc) {
                        d[idx] = b;
                        d[ixj] = a;
                    }
                }
            }
            __syncthreads();
        }
    }
    if (P <= SORT_SMEM)
        for (ll k = threadIdx.x; k < cnt; k += SORT_BLOCK) keys[k] = s[k];
}

__global__ void __launch_bounds__(SORT_BLOCK) k_sort_events(DevCtl *ctl, ull *keys, ll cap, int radix_follows)
{
    sort_events(ctl, keys, cap, radix_follows);
}

/* ------------------------------------------------------------------------ */
/* K8: fragment emission (fragcalc.go:94-117)                               */
/* ------------------------------------------------------------------------ */

__device__ static void frag_emit(const BodyArrays &A, const BodyArrays &F, DevCtl *ctl, ll blk, const ll *blk_off)
{
    const ll n = ctl->n;
    const ll base = blk * NBG_SCAN_TILE;
    if (base >= n) return;
    ll c[NBG_SCAN_ITEMS];
    ll s = 0;
    for (int q = 0; q < NBG_SCAN_ITEMS; q++) {
        ll k = base + (ll)threadIdx.x * NBG_SCAN_ITEMS + q;
        c[q] = k < n ? frag_emit_count(A, k) : 0;
        s += c[q];
    }
    ll tot;
    ll off = block_excl_scan(s, &tot) + blk_off[blk];
    const ll id0 = ctl->next_id;
    const ull seed = ctl->seed, cycle = ctl->cycle;
    for (int q = 0; q < NBG_SCAN_ITEMS; q++) {
        ll k = base + (ll)threadIdx.x * NBG_SCAN_ITEMS + q;
        if (k >= n) break;
        unsigned fk = A.flags[k];
        if ((fk & NBG_LIVE_MASK) != NBG_LIVE_MASK) continue;
        /* for (; fragments > 0;) { fragments--; emit; cnt++; if cnt > 100 break } */
        const ll parent = A.id[k];
        const ull key = nbg_frag_key(seed, parent, cycle);
        const double cx = A.fr_cx[k], cy = A.fr_cy[k], cz = A.fr_cz[k];
        const double rad9 = A.fr_rad[k] * .9;
        for (ll e = 0; e < c[q]; e++) {
            double px, py, pz;
            nbg_frag_point(key, (int)e, cx, cy, cz, rad9, &px, &py, &pz);
            const ll slot = off + e;
            F.id[slot] = id0 + slot;
            F.x[slot] = px;
            F.y[slot] = py;
            F.z[slot] = pz;
            F.vx[slot] = A.vx[k];
            F.vy[slot] = A.vy[k];
            F.vz[slot] = A.vz[k];
            F.m[slot] = A.fr_mass[k];
            F.rad[slot] = A.fr_newrad[k];
            F.fx[slot] = 0;
            F.fy[slot] = 0;
            F.fz[slot] = 0;
            F.ff[slot] = 0;
            F.fs[slot] = 0;
            F.rest[slot] = 0;
            F.fr_rad[slot] = 0;
            F.fr_newrad[slot] = 0;
            F.fr_mass[slot] = 0;
            F.fr_cx[slot] = 0;
            F.fr_cy[slot] = 0;
            F.fr_cz[slot] = 0;
            F.fr_cnt[slot] = 0;
            F.flags[slot] = NBG_F_EXISTS | ((unsigned)NBG_ELASTIC << NBG_BEHAVIOR_SHIFT);
        }
        off += c[q];
        ll left = A.fr_cnt[k] - c[q];
        A.fr_cnt[k] = left;
        if (left <= 0) A.flags[k] = fk & ~NBG_F_EXISTS;
    }
}

__global__ void __launch_bounds__(NBG_SCAN_BLOCK) k_frag_emit(BodyArrays A, BodyArrays F, DevCtl *ctl, const ll *blk_off)
{
    if (ctl->error) return;
    frag_emit(A, F, ctl, blockIdx.x, blk_off);
}

/* both for a collection of one scan tile's capacity */
static_assert(SORT_BLOCK == NBG_SCAN_BLOCK, "one block does both");
__global__ void __launch_bounds__(NBG_SCAN_BLOCK) k_events_small(BodyArrays A, BodyArrays F, DevCtl *ctl, ull *keys,
                                                                 ll ev_cap, const ll *blk_off)
{
    sort_events(ctl, keys, ev_cap, 0);
    __syncthreads();
    if (ctl->error) return;
    frag_emit(A, F, ctl, 0, blk_off);
}

/* ------------------------------------------------------------------------ */
/* K5: collision resolution, newest event first, a thread or a warp to one  */
/* ------------------------------------------------------------------------ */

struct ElasticOut {
    bool collided;
    double vx1, vy1, vz1, vx2, vy2, vz2, vx_cm, vy_cm, vz_cm;
};

/* calcElasticCollision, collisioncalc.go:42-186 (coll3d), on bodies b and o. */
__device__ static ElasticOut elastic_calc(const BodyArrays &A, ll b, ll o)
{
    ElasticOut res;
    res.collided = false;
    res.vx1 = res.vy1 = res.vz1 = res.vx2 = res.vy2 = res.vz2 = 0;
    res.vx_cm = res.vy_cm = res.vz_cm = 0;
    const double m1 = A.m[b], m2 = A.m[o], r1 = A.rad[b], r2 = A.rad[o];
    const double x1 = A.x[b], y1 = A.y[b], z1 = A.z[b];
    const double X2 = A.x[o], Y2 = A.y[o], Z2 = A.z[o];
    const double ux1 = A.vx[b], uy1 = A.vy[b], uz1 = A.vz[b];
    const double vx2 = A.vx[o], vy2 = A.vy[o], vz2 = A.vz[o];

    const double r12 = r1 + r2;
    const double m21 = m2 / m1;
    const double x21 = X2 - x1, y21 = Y2 - y1, z21 = Z2 - z1;
    const double vx21 = vx2 - ux1, vy21 = vy2 - uy1, vz21 = vz2 - uz1;
    const double vx_cm = (m1 * ux1 + m2 * vx2) / (m1 + m2);
    const double vy_cm = (m1 * uy1 + m2 * vy2) / (m1 + m2);
    const double vz_cm = (m1 * uz1 + m2 * vz2) / (m1 + m2);
    const double d = sqrt(x21 * x21 + y21 * y21 + z21 * z21);
    const double v = sqrt(vx21 * vx21 + vy21 * vy21 + vz21 * vz21);
    if (v == 0) return res;
    /* ball 1 at the origin, ball 2 at rest */
    const double px = x21, py = y21, pz = z21;
    const double wx = -vx21, wy = -vy21, wz = -vz21;
    const double theta2 = nbg_acos(pz / d);
    const double phi2 = (px == 0 && py == 0) ? 0.0 : nbg_atan2(py, px);
    const double st = nbg_sin(theta2), ct = nbg_cos(theta2);
    const double sp = nbg_sin(phi2), cp = nbg_cos(phi2);
    double vx1r = ct * cp * wx + ct * sp * wy - st * wz;
    double vy1r = cp * wy - sp * wx;
    double vz1r = st * cp * wx + st * sp * wy + ct * wz;
    double fvz1r = vz1r / v;
    if (fvz1r > 1)
        fvz1r = 1;
    else if (fvz1r < -1)
        fvz1r = -1;
    const double thetav = nbg_acos(fvz1r);
    const double phiv = (vx1r == 0 && vy1r == 0) ? 0.0 : nbg_atan2(vy1r, vx1r);
    const double dr = d * nbg_sin(thetav) / r12;
    if (thetav > NBG_PIO2_HI || fabs(dr) > 1) return res;
    const double alpha = nbg_asin(-dr);
    const double beta = phiv;
    const double sbeta = nbg_sin(beta), cbeta = nbg_cos(beta);
    const double a = nbg_tan(thetav + alpha);
    const double dvz2 = 2 * (vz1r + a * (cbeta * vx1r + sbeta * vy1r)) / ((1 + a * a) * (1 + m21));
    const double vz2r = dvz2;
    const double vx2r = a * cbeta * dvz2;
    const double vy2r = a * sbeta * dvz2;
    vz1r = vz1r - m21 * vz2r;
    vx1r = vx1r - m21 * vx2r;
    vy1r = vy1r - m21 * vy2r;
    res.collided = true;
    res.vx1 = ct * cp * vx1r - sp * vy1r + st * cp * vz1r + vx2;
    res.vy1 = ct * sp * vx1r + cp * vy1r + st * sp * vz1r + vy2;
    res.vz1 = ct * vz1r - st * vx1r + vz2;
    res.vx2 = ct * cp * vx2r - sp * vy2r + st * cp * vz2r + vx2;
    res.vy2 = ct * sp * vx2r + cp * vy2r + st * sp * vz2r + vy2;
    res.vz2 = ct * vz2r - st * vx2r + vz2;
    res.vx_cm = vx_cm;
    res.vy_cm = vy_cm;
    res.vz_cm = vz_cm;
    return res;
}

/* initiateFragmentation, fragcalc.go:67-85.  newRadius is always 1: Go
 * evaluates the exponent 1/3 as integer division (0) and Pow(x, 0) == 1. */
__device__ static void initiate_frag(BodyArrays &A, ll b, double fragFactor)
{
    const double ffb = A.ff[b];
    const double fragDelta = ffb > 10 ? 10.0 : fragFactor - ffb;
    const double fragments = nbg_go_min(fragDelta * A.fs[b], NBG_MAX_FRAGS);
    unsigned f = A.flags[b];
    if (fragments <= 1) {
        A.flags[b] = (f & ~(3u << NBG_BEHAVIOR_SHIFT)) | ((unsigned)NBG_FRAGMENT << NBG_BEHAVIOR_SHIFT);
        return;
    }
    A.flags[b] = f | NBG_F_FRAGMENTING;
    A.fr_rad[b] = A.rad[b];
    A.fr_newrad[b] = 1.0;
    A.fr_mass[b] = A.m[b] / fragments;
    A.fr_cnt[b] = fragments != fragments ? 0 : (ll)fragments; /* int(NaN): no fragment either way */
    A.fr_cx[b] = A.x[b];
    A.fr_cy[b] = A.y[b];
    A.fr_cz[b] = A.z[b];
}

/* whether ResolveCollision goes on to the elastic formulas */
__device__ static bool collision_resolves(const BodyArrays &A, ll b, ll o)
{
    const unsigned fb = A.flags[b], fo = A.flags[o];
    if (!(fb & NBG_F_EXISTS) || !(fo & NBG_F_EXISTS)) return false;
    const unsigned bb = NBG_BEHAVIOR(fb), bo = NBG_BEHAVIOR(fo);
    return bb == NBG_ELASTIC && (bo == NBG_ELASTIC || bo == NBG_FRAGMENT);
}

/* What becomes of bodies b and o, given their velocities after the collision
 * (restitution applied): shouldFragment / doFragment / doElastic
 * (fragcalc.go:24-61, collisioncalc.go:26-35). */
__device__ static __noinline__ void apply_collision(BodyArrays &A, ll b, ll o, double nvx1, double nvy1, double nvz1, double nvx2,
                                       double nvy2, double nvz2)
{
    const unsigned bb = NBG_BEHAVIOR(A.flags[b]), bo = NBG_BEHAVIOR(A.flags[o]);
    bool frag = false;
    double tf = 0, of = 0;
    if (bb == NBG_FRAGMENT || bo == NBG_FRAGMENT) {
        const double vThis = A.vx[b] + A.vy[b] + A.vz[b];
        const double dvThis = fabs(A.vx[b] - nvx1) + fabs(A.vy[b] - nvy1) + fabs(A.vz[b] - nvz1);
        const double thisFactor = dvThis / fabs(vThis);
        const double vOther = A.vx[o] + A.vy[o] + A.vz[o];
        const double dvOther = fabs(A.vx[o] - nvx2) + fabs(A.vy[o] - nvy2) + fabs(A.vz[o] - nvz2);
        const double otherFactor = dvOther / fabs(vOther);
        if ((bb == NBG_FRAGMENT && thisFactor > A.ff[b]) || (bo == NBG_FRAGMENT && otherFactor > A.ff[o])) {
            frag = true;
            tf = thisFactor;
            of = otherFactor;
        }
    }
    if (frag) {
        if (bb == NBG_FRAGMENT && tf > A.ff[b]) initiate_frag(A, b, tf);
        if (NBG_BEHAVIOR(A.flags[o]) == NBG_FRAGMENT && of > A.ff[o]) initiate_frag(A, o, of);
        return;
    }
    A.vx[b] = nvx1;
    A.vy[b] = nvy1;
    A.vz[b] = nvz1;
    A.vx[o] = nvx2;
    A.vy[o] = nvy2;
    A.vz[o] = nvz2;
    A.flags[b] |= NBG_F_COLLIDED;
    A.flags[o] |= NBG_F_COLLIDED;
}

/* ResolveCollision, body.go:248-264 */
__device__ static void resolve_collision(BodyArrays &A, ll b, ll o)
{
    if (!collision_resolves(A, b, o)) return;
    const ElasticOut r = elastic_calc(A, b, o);
    if (!r.collided) return;
    const double rb = A.rest[b];
    apply_collision(A, b, o, (r.vx1 - r.vx_cm) * rb + r.vx_cm, (r.vy1 - r.vy_cm) * rb + r.vy_cm,
                    (r.vz1 - r.vz_cm) * rb + r.vz_cm, (r.vx2 - r.vx_cm) * rb + r.vx_cm,
                    (r.vy2 - r.vy_cm) * rb + r.vy_cm, (r.vz2 - r.vz_cm) * rb + r.vz_cm);
}

/* ---- one collision by a whole warp ------------------------------------------
 * An FP64 operation takes 64 cycles however many lanes it serves, and the
 * formulas are a chain of about 1,100 of them.  Where few
 * events can be resolved at once, a warp takes one: its lanes evaluate the two
 * angles of a direction, the sines and cosines of both, the quotients and the
 * components side by side, through the same operations in the same order (a
 * coefficient or operand chosen by lane in place of a branch), so the results
 * are the same bit for bit.  Two events on one pair of bodies, the usual cycle of
 * a 1,000-body disk: 81 -> 40 us under the profiler, caches cold, of which most is
 * then fetching the code, and 18 us off a cycle of 143. */
__device__ __forceinline__ double lane_of(double v, int src) { return __shfl_sync(0xffffffffu, v, src); }

/* Out of line, the functions that follow: the code runs once a cycle, so what
 * fetching it costs counts. */
__device__ static __noinline__ double lane_div(double a, double b) { return a / b; }
__device__ static __noinline__ double lane_sqrt(double a) { return sqrt(a); }
__device__ static __noinline__ double rare_atan2(double y, double x) { return nbg_atan2(y, x); }

/* nbg_atan2, each lane its own */
__device__ static __noinline__ double lane_atan2(double y, double x)
{
    const double ax = fabs(x), ay = fabs(y);
    if (!(ax > 0.0 && ay > 0.0 && ax <= NBG_DBL_MAX && ay <= NBG_DBL_MAX)) return rare_atan2(y, x);
    const bool swap = !(ay <= ax);
    const double t = lane_div(swap ? ax : ay, swap ? ay : ax);
    const bool big = t > NBG_TAN_PI_12;
    const double u = lane_div(big ? t * NBG_SQRT3 - 1.0 : t, big ? t + NBG_SQRT3 : 1.0);
    const double p = nbg_atan_poly(u);
    const double a = big ? NBG_PIO6_HI + (p + NBG_PIO6_LO) : p;
    double r = swap ? NBG_PIO2_HI - (a - NBG_PIO2_LO) : a;
    if (x < 0.0) r = NBG_PI_HI - (r - NBG_PI_LO);
    return copysign(r, y);
}

/* nbg_sin_poly or nbg_cos_poly, chosen by lane */
__device__ static __noinline__ double lane_poly(double r, bool c)
{
    const double z = r * r;
    double p = c ? NBG_C11 : NBG_S10;
    p = (c ? NBG_C10 : NBG_S9) + z * p;
    p = (c ? NBG_C9 : NBG_S8) + z * p;
    p = (c ? NBG_C8 : NBG_S7) + z * p;
    p = (c ? NBG_C7 : NBG_S6) + z * p;
    p = (c ? NBG_C6 : NBG_S5) + z * p;
    p = (c ? NBG_C5 : NBG_S4) + z * p;
    p = (c ? NBG_C4 : NBG_S3) + z * p;
    p = (c ? NBG_C3 : NBG_S2) + z * p;
    p = (c ? NBG_C2 : NBG_S1) + z * p;
    const double m = (c ? z : r) * z * p; /* the term that the polynomial makes */
    if (!c) return r + m;
    const double hz = 0.5 * z;
    const double w = 1.0 - hz;
    return w + (((1.0 - w) - hz) + m);
}

/* nbg_sin or nbg_cos, chosen by lane */
__device__ static __noinline__ double lane_sincos(double x, bool c)
{
    if (!nbg_isfinite(x)) return nbg_nan();
    if (x == 0.0 && !c) return x;
    int q;
    const double r = nbg_reduce_pio2(x, &q);
    const double v = lane_poly(r, c != ((q & 1) != 0));
    return (c ? q == 1 || q == 2 : q >= 2) ? -v : v;
}

/* resolve_collision; b and o the same in every lane */
__device__ static __noinline__ void resolve_collision_warp(BodyArrays &A, ll b, ll o)
{
    if (!collision_resolves(A, b, o)) return;
    const int lane = threadIdx.x & 31;
    const double m1 = A.m[b], m2 = A.m[o], r1 = A.rad[b], r2 = A.rad[o];
    const double x1 = A.x[b], y1 = A.y[b], z1 = A.z[b];
    const double X2 = A.x[o], Y2 = A.y[o], Z2 = A.z[o];
    const double ux1 = A.vx[b], uy1 = A.vy[b], uz1 = A.vz[b];
    const double vx2 = A.vx[o], vy2 = A.vy[o], vz2 = A.vz[o];
    const double rb = A.rest[b];
    __syncwarp();

    const double r12 = r1 + r2;
    const double x21 = X2 - x1, y21 = Y2 - y1, z21 = Z2 - z1;
    const double vx21 = vx2 - ux1, vy21 = vy2 - uy1, vz21 = vz2 - uz1;
    /* lane 0: m21; lanes 1 to 3: the centre's velocity */
    const double u = lane == 1 ? ux1 : lane == 2 ? uy1 : uz1, w2 = lane == 1 ? vx2 : lane == 2 ? vy2 : vz2;
    const double quot = lane_div(lane == 0 ? m2 : m1 * u + m2 * w2, lane == 0 ? m1 : m1 + m2);
    const double m21 = lane_of(quot, 0);
    /* lane 0: the distance; lane 1: the relative speed */
    const double e1 = lane == 0 ? x21 : vx21, e2 = lane == 0 ? y21 : vy21, e3 = lane == 0 ? z21 : vz21;
    const double len = lane_sqrt(e1 * e1 + e2 * e2 + e3 * e3);
    const double d = lane_of(len, 0), v = lane_of(len, 1);
    if (v == 0) return;
    const double px = x21, py = y21, pz = z21;
    const double wx = -vx21, wy = -vy21, wz = -vz21;

    /* lane 0: an acos as nbg_acos(t) evaluates it; lane 1: an atan2, 0 at
     * the origin */
    auto angles = [&](double t, double y, double x) {
        const double s = lane_sqrt((1.0 - t) * (1.0 + t));
        double a = lane_atan2(lane == 0 ? s : y, lane == 0 ? t : x);
        if (lane == 0 && !(fabs(t) <= 1.0)) a = t != t ? t + t : nbg_nan();
        if (lane != 0 && x == 0 && y == 0) a = 0.0;
        return a;
    };
    const double a2 = angles(lane_div(pz, d), py, px);
    const double theta2 = lane_of(a2, 0), phi2 = lane_of(a2, 1);
    const double sc = lane_sincos(lane < 2 ? theta2 : phi2, lane & 1);
    const double st = lane_of(sc, 0), ct = lane_of(sc, 1), sp = lane_of(sc, 2), cp = lane_of(sc, 3);
    /* lane 0: vx1r; lane 1: vz1r */
    const double P = lane == 0 ? ct : st, Q = lane == 0 ? -st : ct;
    const double vr = P * cp * wx + P * sp * wy + Q * wz;
    double vx1r = lane_of(vr, 0), vz1r = lane_of(vr, 1);
    double vy1r = cp * wy - sp * wx;
    double fvz1r = lane_div(vz1r, v);
    if (fvz1r > 1)
        fvz1r = 1;
    else if (fvz1r < -1)
        fvz1r = -1;
    const double av = angles(fvz1r, vy1r, vx1r);
    const double thetav = lane_of(av, 0), beta = lane_of(av, 1);
    /* lane 0: sin thetav; lanes 2 and 3: sine and cosine of beta */
    const double sv = lane_sincos(lane < 2 ? thetav : beta, lane & 1);
    const double sbeta = lane_of(sv, 2), cbeta = lane_of(sv, 3);
    const double dr = lane_div(d * lane_of(sv, 0), r12);
    if (thetav > NBG_PIO2_HI || fabs(dr) > 1) return;
    /* nbg_asin(-dr); it is not above 1 in magnitude, but may be NaN */
    const double alpha = dr != dr ? -dr + -dr : lane_atan2(-dr, lane_sqrt((1.0 - -dr) * (1.0 + -dr)));
    const double ta = thetav + alpha;
    double a;
    if (ta == 0.0) {
        a = ta;
    } else if (!nbg_isfinite(ta)) {
        a = nbg_nan();
    } else {
        int q;
        const double r = nbg_reduce_pio2(ta, &q);
        const double pl = lane_poly(r, lane & 1);
        const double ps = lane_of(pl, 0), pc = lane_of(pl, 1);
        a = lane_div((q & 1) ? -pc : ps, (q & 1) ? ps : pc);
    }
    const double dvz2 = lane_div(2 * (vz1r + a * (cbeta * vx1r + sbeta * vy1r)), (1 + a * a) * (1 + m21));
    const double vz2r = dvz2;
    const double vx2r = a * cbeta * dvz2;
    const double vy2r = a * sbeta * dvz2;
    vz1r = vz1r - m21 * vz2r;
    vx1r = vx1r - m21 * vx2r;
    vy1r = vy1r - m21 * vy2r;
    /* lanes 0 to 2: components of the first body, 3 to 5: of the second */
    const bool two = lane >= 3;
    const int c = two ? lane - 3 : lane;
    const double X = two ? vx2r : vx1r, Y = two ? vy2r : vy1r, Z = two ? vz2r : vz1r;
    const double S = c == 0 ? cp : sp;
    const double xy = c == 2 ? ct * Z + -st * X : ct * S * X + (c == 0 ? -sp : cp) * Y;
    const double xyz = c == 2 ? xy : xy + st * S * Z;
    const double vel = xyz + (c == 0 ? vx2 : c == 1 ? vy2 : vz2);
    const double cm = lane_of(quot, 1 + (lane < 6 ? c : 0));
    const double nv = (vel - cm) * rb + cm;
    const double n0 = lane_of(nv, 0), n1 = lane_of(nv, 1), n2 = lane_of(nv, 2), n3 = lane_of(nv, 3),
                 n4 = lane_of(nv, 4), n5 = lane_of(nv, 5);
    if (lane == 0) apply_collision(A, b, o, n0, n1, n2, n3, n4, n5);
    __syncwarp();
}

/* ResolveSubsume, body.go:228-244 (no Exists checks, radius unchanged). */
__device__ static void resolve_subsume(BodyArrays &A, ll b, ll o)
{
    const double thisMass = A.m[b], otherMass = A.m[o];
    A.m[b] = thisMass + otherMass;
    A.m[o] = 0;
    A.flags[o] &= ~NBG_F_EXISTS;
}

/* first index of sorted keys[0..cnt) that is >= v */
__device__ static ll lower_bound_u64(const ull *keys, ll cnt, ull v)
{
    ll lo = 0, hi = cnt;
    while (lo < hi) {
        const ll mid = (lo + hi) >> 1;
        if (keys[mid] < v)
            lo = mid + 1;
        else
            hi = mid;
    }
    return lo;
}

/* ProcessMods (body_collection.go:213-235): each sim resolves its own events
 * newest first.  Events of one sim only touch that sim's bodies, and the
 * sorted keys are grouped by sim (i ranges).
 *
 * One CTA per sim.  Resolving an event reads and writes only its two bodies,
 * so the sequential order only matters between events that share a body:
 * the CTA resolves in rounds, and in each round every pending event that is
 * the oldest pending one (in processing order) on both of its bodies is
 * resolved, all such events in parallel.  Every body sees its events in the
 * sequential order, so the result is the sequential result bit for bit.
 * owner[] (one word per body; any contents on entry) holds, per round, the
 * smallest pending processing index that touches the body.  Once a round
 * resolves fewer than RESOLVE_MIN_ROUND events (two, among few: a long chain
 * through one body, as when a large body absorbs many), one warp finishes the
 * rest in order.  ev_out holds the sims one after another, each in processing order;
 * its pad field marks pending events during the kernel and is 0 on return. */
#define RESOLVE_BLOCK 256
#define RESOLVE_WARPS (RESOLVE_BLOCK / 32)
#define RESOLVE_MIN_ROUND 8 /* fewer events resolved in a round: finish sequentially */

__device__ static void event_bodies(ull key, ll &b1, ll &b2, unsigned &type)
{
    const ll i = (ll)(key >> 32);
    const ll j = (ll)((key >> 2) & 0x3fffffffull);
    type = (unsigned)(key & 3ull);
    b1 = i;
    b2 = j;
    if (type == NBG_EVT_SUB_JI) {
        b1 = j;
        b2 = i;
    }
}

__device__ static void resolve_one(BodyArrays &A, ull key, nbg_event *out)
{
    ll b1, b2;
    unsigned type;
    event_bodies(key, b1, b2, type);
    nbg_event e;
    e.id1 = A.id[b1];
    e.id2 = A.id[b2];
    e.type = type == NBG_EVT_COLL_IJ ? NBG_EV_COLLISION : NBG_EV_SUBSUME;
    e.pad = 0;
    if (type == NBG_EVT_COLL_IJ)
        resolve_collision(A, b1, b2);
    else
        resolve_subsume(A, b1, b2);
    *out = e;
}

/* the same by a whole warp, the arguments the same in every lane */
__device__ static __noinline__ void resolve_one_warp(BodyArrays &A, ull key, nbg_event *out)
{
    ll b1, b2;
    unsigned type;
    event_bodies(key, b1, b2, type);
    if (type == NBG_EVT_COLL_IJ) resolve_collision_warp(A, b1, b2);
    __syncwarp();
    if ((threadIdx.x & 31) == 0) {
        if (type != NBG_EVT_COLL_IJ) resolve_subsume(A, b1, b2);
        nbg_event e;
        e.id1 = A.id[b1];
        e.id2 = A.id[b2];
        e.type = type == NBG_EVT_COLL_IJ ? NBG_EV_COLLISION : NBG_EV_SUBSUME;
        e.pad = 0;
        *out = e;
    }
    __syncwarp();
}

/* ---- resolution links: the events of a busy cycle in dataflow order ------
 * ProcessMods resolves events one after another, newest first.  Two events
 * that share no body commute, so an event may be resolved as soon as every
 * earlier event on each of its bodies is: the per-body chains of events in
 * processing order are the only order that matters.  For cycles with more
 * events than the one-block sort holds, the chains are built from the sorted
 * (body, event) incidences, and k_resolve works through the ready events
 * round by round, touching only those - the result is the sequential one
 * bit for bit, however many events resolve at once. */

__device__ __forceinline__ bool links_on(const DevCtl *ctl)
{
    return ctl->error == 0 && ctl->ev_count > NBG_EV_BLOCK_SORT;
}

/* sim s holds the sorted events [ev_lo[s], ev_lo[s + 1]) */
__global__ void k_ev_ranges(DevCtl *ctl, SimSegs seg, const ull *keys, ll *ev_lo)
{
    if (!links_on(ctl)) return;
    const ll cnt = ctl->ev_count;
    for (int s = blockIdx.x * blockDim.x + threadIdx.x; s <= seg.nsims; s += gridDim.x * blockDim.x)
        ev_lo[s] = s == seg.nsims ? cnt : (s == 0 ? 0 : lower_bound_u64(keys, cnt, (ull)seg.off[s] << 32));
}

/* The two incidences of the event at sorted position t, processing index o
 * (its sim's events in reverse key order): body << (ob + 1) | o << 1 | side */
__global__ void k_ev_incid(DevCtl *ctl, SimSegs seg, const ull *keys, const ll *ev_lo, ull *inc, int ob)
{
    if (!links_on(ctl)) return;
    const ll cnt = ctl->ev_count;
    for (ll t = (ll)blockIdx.x * blockDim.x + threadIdx.x; t < cnt; t += (ll)gridDim.x * blockDim.x) {
        const ull key = keys[t];
        ll b1, b2;
        unsigned ty;
        event_bodies(key, b1, b2, ty);
        const int s = seg.nsims == 1 ? 0 : nbg_sim_of(seg.off, seg.nsims, (ll)(key >> 32));
        const ull o = (ull)(ev_lo[s] + ev_lo[s + 1] - 1 - t);
        inc[2 * t] = ((ull)b1 << (ob + 1)) | (o << 1);
        inc[2 * t + 1] = ((ull)b2 << (ob + 1)) | (o << 1) | 1ull;
    }
}

/* From the sorted incidences: each event's next event on each of its bodies
 * (link[2 o + side], -1: none) and previous one (pred[2 o + side]). */
__global__ void k_ev_links(DevCtl *ctl, const ull *inc, int ob, ll *link, ll *pred)
{
    if (!links_on(ctl)) return;
    const ll m2 = 2 * ctl->ev_count;
    const ull omask = (1ull << ob) - 1ull;
    for (ll t = (ll)blockIdx.x * blockDim.x + threadIdx.x; t < m2; t += (ll)gridDim.x * blockDim.x) {
        const ull k = inc[t];
        const ull b = k >> (ob + 1);
        const ll slot = 2 * (ll)((k >> 1) & omask) + (ll)(k & 1ull);
        link[slot] = t + 1 < m2 && (inc[t + 1] >> (ob + 1)) == b ? (ll)((inc[t + 1] >> 1) & omask) : -1;
        pred[slot] = t > 0 && (inc[t - 1] >> (ob + 1)) == b ? (ll)((inc[t - 1] >> 1) & omask) : -1;
    }
}

/* unresolved predecessors of each event: one per body, once if both bodies'
 * previous event is the same */
__global__ void k_ev_pending(DevCtl *ctl, const ll *pred, int *pend)
{
    if (!links_on(ctl)) return;
    const ll m = ctl->ev_count;
    for (ll o = (ll)blockIdx.x * blockDim.x + threadIdx.x; o < m; o += (ll)gridDim.x * blockDim.x) {
        const ll p0 = pred[2 * o], p1 = pred[2 * o + 1];
        pend[o] = (p0 >= 0 ? 1 : 0) + (p1 >= 0 && p1 != p0 ? 1 : 0);
    }
}

/* Resolution of one sim's events through its links: round by round, every
 * ready event (all earlier events on its bodies resolved) at once. */
__device__ static void resolve_dataflow(BodyArrays &A, DevCtl *ctl, const ull *keys, nbg_event *ev_out, ll lo, ll hi,
                                        const ll *link, int *pend, ll *front, ll ev_cap)
{
    __shared__ ll s_n[2];
    __shared__ ll s_total;
    const int tid = threadIdx.x;
    ll *fr[2] = {front + lo, front + ev_cap + lo};
    if (tid == 0) {
        s_n[0] = s_n[1] = 0;
        s_total = 0;
    }
    __syncthreads();
    for (ll o = lo + tid; o < hi; o += RESOLVE_BLOCK)
        if (pend[o] == 0) fr[0][atomicAdd((unsigned long long *)&s_n[0], 1ull)] = o;
    __syncthreads();
    int cur = 0;
    ll done = 0;
    while (s_n[cur] > 0) {
        const ll nr = s_n[cur];
        if (nr == 1) {
            /* a chain (one body in every event): one thread follows it for
             * as long as each event readies exactly one successor, without
             * a barrier per event */
            if (tid == 0) {
                ll o = fr[cur][0];
                for (;;) {
                    resolve_one(A, keys[lo + hi - 1 - o], &ev_out[o]);
                    done++;
                    const ll n0 = link[2 * o], n1 = link[2 * o + 1];
                    ll rd[2];
                    int nready = 0;
                    if (n0 >= 0 && atomicSub(&pend[n0], 1) == 1) rd[nready++] = n0;
                    if (n1 >= 0 && n1 != n0 && atomicSub(&pend[n1], 1) == 1) rd[nready++] = n1;
                    if (nready == 1) {
                        o = rd[0];
                        continue;
                    }
                    for (int q = 0; q < nready; q++) fr[cur ^ 1][s_n[cur ^ 1]++] = rd[q];
                    break;
                }
            }
        } else
        for (ll x = tid; x < nr; x += RESOLVE_BLOCK) {
            const ll o = fr[cur][x];
            resolve_one(A, keys[lo + hi - 1 - o], &ev_out[o]);
            done++;
            const ll n0 = link[2 * o], n1 = link[2 * o + 1];
            if (n0 >= 0 && atomicSub(&pend[n0], 1) == 1)
                fr[cur ^ 1][atomicAdd((unsigned long long *)&s_n[cur ^ 1], 1ull)] = n0;
            if (n1 >= 0 && n1 != n0 && atomicSub(&pend[n1], 1) == 1)
                fr[cur ^ 1][atomicAdd((unsigned long long *)&s_n[cur ^ 1], 1ull)] = n1;
        }
        __syncthreads(); /* this round's bodies are written, the next frontier complete */
        if (tid == 0) s_n[cur] = 0;
        cur ^= 1;
        __syncthreads();
    }
    atomicAdd((unsigned long long *)&s_total, (ull)done);
    __syncthreads();
    /* every event has a chain of predecessors back to a ready one, so all
     * resolve; anything else is a broken invariant, reported as such */
    if (tid == 0 && s_total != (ull)(hi - lo)) {
        ctl->error = NBG_E_STATE;
        ctl->error_what = 7;
        ctl->error_need = hi - lo - (ll)s_total;
    }
}

__global__ void __launch_bounds__(RESOLVE_BLOCK) k_resolve(BodyArrays A, DevCtl *ctl, SimSegs seg, const ull *keys,
                                                           nbg_event *ev_out, unsigned *owner, int links,
                                                           const ll *ev_lo, const ll *link, int *pend, ll *front,
                                                           ll ev_cap)
{
    __shared__ int s_left, s_done, s_ready;
    __shared__ ll s_first[RESOLVE_WARPS];
    if (ctl->error) return;
    const ll cnt = ctl->ev_count;
    const int s = blockIdx.x;
    const int tid = threadIdx.x;
    if (s == 0 && tid == 0) {
        ctl->next_id += ctl->frag_total; /* fragments took ids next_id .. next_id+total-1 */
        ctl->last_ev_n = cnt;
        ctl->acc_events += cnt;
        ctl->acc_frags += ctl->frag_total;
    }
    if (s >= seg.nsims) return;
    if (links && cnt > NBG_EV_BLOCK_SORT) {
        const ll lo = ev_lo[s], hi = ev_lo[s + 1];
        if (hi > lo) resolve_dataflow(A, ctl, keys, ev_out, lo, hi, link, pend, front, ev_cap);
        return;
    }
    const ll lo = seg.nsims == 1 ? 0 : lower_bound_u64(keys, cnt, (ull)seg.off[s] << 32);
    const ll hi = seg.nsims == 1 ? cnt : lower_bound_u64(keys, cnt, (ull)seg.off[s + 1] << 32);
    const ll m = hi - lo;
    if (m <= 0) return;
    if (m == 1) {
        if (tid < 32) resolve_one_warp(A, keys[lo], &ev_out[lo]);
        return;
    }
    /* processing index p is keys[hi - 1 - p], written to ev_out[lo + p] */
    for (ll p = tid; p < m; p += RESOLVE_BLOCK) ev_out[lo + p].pad = 1;
    if (tid == 0) s_left = (int)(m < 0x7fffffff ? m : 0x7fffffff);
    __syncthreads();
    for (ll round = 0; round < m; round++) {
        for (ll p = tid; p < m; p += RESOLVE_BLOCK) {
            if (ev_out[lo + p].pad) {
                ll b1, b2;
                unsigned ty;
                event_bodies(keys[hi - 1 - p], b1, b2, ty);
                owner[b1] = 0xffffffffu;
                owner[b2] = 0xffffffffu;
            }
        }
        __syncthreads();
        for (ll p = tid; p < m; p += RESOLVE_BLOCK) {
            if (ev_out[lo + p].pad) {
                ll b1, b2;
                unsigned ty;
                event_bodies(keys[hi - 1 - p], b1, b2, ty);
                atomicMin(&owner[b1], (unsigned)p);
                atomicMin(&owner[b2], (unsigned)p);
            }
        }
        if (tid == 0) s_done = s_ready = 0;
        __syncthreads();
        auto ready = [&](ll p) {
            if (!ev_out[lo + p].pad) return false;
            ll b1, b2;
            unsigned ty;
            event_bodies(keys[hi - 1 - p], b1, b2, ty);
            return owner[b1] == (unsigned)p && owner[b2] == (unsigned)p;
        };
        for (ll p = tid; p < m; p += RESOLVE_BLOCK)
            if (ready(p)) {
                const int k = atomicAdd(&s_ready, 1);
                if (k < RESOLVE_WARPS) s_first[k] = p;
            }
        __syncthreads();
        if (s_ready <= RESOLVE_WARPS) {
            /* few: a warp to each */
            if ((tid >> 5) < s_ready) {
                const ll p = s_first[tid >> 5];
                resolve_one_warp(A, keys[hi - 1 - p], &ev_out[lo + p]);
            }
            if (tid == 0) s_done = s_ready;
        } else {
            int done = 0;
            for (ll p = tid; p < m; p += RESOLVE_BLOCK)
                if (ready(p)) {
                    resolve_one(A, keys[hi - 1 - p], &ev_out[lo + p]); /* clears pad */
                    done++;
                }
            if (done) atomicAdd(&s_done, done);
        }
        __syncthreads();
        if (tid == 0) s_left -= s_done;
        __syncthreads();
        if (s_left <= 0) return;
        /* a chain of events on shared bodies: a round no longer pays for
         * itself (one over few events is a few barriers, less than an event) */
        if (s_done < (m <= RESOLVE_BLOCK ? 2 : RESOLVE_MIN_ROUND)) break;
    }
    /* the rest in processing order, one warp: every pending event's
     * predecessors are resolved or come before it */
    if (tid < 32)
        for (ll p = 0; p < m; p++)
            if (ev_out[lo + p].pad) resolve_one_warp(A, keys[hi - 1 - p], &ev_out[lo + p]);
}

/* ------------------------------------------------------------------------ */
/* K6: integration (Update, body.go:114-139) + renderables                 */
/* ------------------------------------------------------------------------ */

__global__ void k_integrate(BodyArrays A, DevCtl *ctl, nbg_renderable *rend, nbg_renderable *ring_rend, ll ring_cap,
                            int ring_slots)
{
    if (ctl->error) return;
    const ll n = ctl->n;
    const double dt = ctl->dt, R = ctl->R;
    ll nan_local = 0;
    /* this cycle's slot of the render ring, if one is attached */
    nbg_renderable *ring = ring_rend ? ring_rend + (ll)(ctl->cycle % (ull)ring_slots) * ring_cap : nullptr;
    for (ll k = (ll)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += (ll)gridDim.x * blockDim.x) {
        unsigned f = A.flags[k];
        nbg_renderable r;
        r.id = A.id[k];
        if (!(f & NBG_F_EXISTS)) {
            r.x = r.y = r.z = 0.0f;
            r.flags = 0;
            r.radius = 0.0;
            rend[k] = r;
            if (ring && k < ring_cap) ring[k] = r;
            continue;
        }
        double vx = A.vx[k], vy = A.vy[k], vz = A.vz[k];
        if (!(f & NBG_F_COLLIDED)) {
            const double m = A.m[k];
            vx += dt * A.fx[k] / m;
            vy += dt * A.fy[k] / m;
            vz += dt * A.fz[k] / m;
            A.vx[k] = vx;
            A.vy[k] = vy;
            A.vz[k] = vz;
        }
        const double x = A.x[k] + dt * vx;
        const double y = A.y[k] + dt * vy;
        const double z = A.z[k] + dt * vz;
        A.x[k] = x;
        A.y[k] = y;
        A.z[k] = z;
        A.rest[k] = R;
        f &= ~NBG_F_COLLIDED;
        if (x != x || y != y || z != z) {
            f &= ~NBG_F_EXISTS;
            nan_local++;
        }
        A.flags[k] = f;
        r.x = (float)x;
        r.y = (float)y;
        r.z = (float)z;
        r.flags = f & (NBG_F_EXISTS | NBG_F_IS_SUN);
        r.radius = A.rad[k];
        if (!(f & NBG_F_EXISTS)) {
            r.x = r.y = r.z = 0.0f;
            r.flags = 0;
            r.radius = 0.0;
        }
        rend[k] = r;
        if (ring && k < ring_cap) ring[k] = r;
    }
    if (ring) __threadfence_system(); /* the slot's renderables before its header */
    if (nan_local) atomicAdd((unsigned long long *)&ctl->acc_nan, (ull)nan_local);
}

/* the header of this cycle's ring slot, after its renderables: count and
 * written, a system-wide fence, then the cycle */
__global__ void k_ring_header(DevCtl *ctl, nbg_ring_slot *head, ll ring_cap, int ring_slots)
{
    if (ctl->error) return;
    const ull cycle = ctl->cycle;
    const ll n = ctl->n;
    volatile nbg_ring_slot *h = head + cycle % (ull)ring_slots;
    __threadfence_system();
    h->count = n;
    h->written = n < ring_cap ? n : ring_cap;
    __threadfence_system();
    h->cycle = (ll)cycle;
    __threadfence_system();
}

/* ------------------------------------------------------------------------ */
/* K7: Cycle (body_collection.go:253-296): stable compaction + adds         */
/* ------------------------------------------------------------------------ */

__device__ static void copy_body(const BodyArrays &S, ll s, const BodyArrays &D, ll d)
{
    D.x[d] = S.x[s];
    D.y[d] = S.y[s];
    D.z[d] = S.z[s];
    D.vx[d] = S.vx[s];
    D.vy[d] = S.vy[s];
    D.vz[d] = S.vz[s];
    D.m[d] = S.m[s];
    D.rad[d] = S.rad[s];
    D.fx[d] = S.fx[s];
    D.fy[d] = S.fy[s];
    D.fz[d] = S.fz[s];
    D.ff[d] = S.ff[s];
    D.fs[d] = S.fs[s];
    D.rest[d] = S.rest[s];
    D.fr_rad[d] = S.fr_rad[s];
    D.fr_newrad[d] = S.fr_newrad[s];
    D.fr_mass[d] = S.fr_mass[s];
    D.fr_cx[d] = S.fr_cx[s];
    D.fr_cy[d] = S.fr_cy[s];
    D.fr_cz[d] = S.fr_cz[s];
    D.fr_cnt[d] = S.fr_cnt[s];
    D.id[d] = S.id[s];
    D.flags[d] = S.flags[s];
}

__device__ static bool cycle_changes(const DevCtl *ctl)
{
    return ctl->n_keep != ctl->n || ctl->frag_total > 0 || ctl->n_host_adds > 0;
}

/* Kept body k of sim s goes to new_off[s] + (its rank among kept bodies -
 * keep_start[s]): the order inside each sim is preserved. */
#define NBG_GONE 0xffffffffu

__device__ static void compact(const BodyArrays &A, const BodyArrays &Bt, const DevCtl *ctl, const SimSegs &seg, ll blk,
                               const ll *blk_off, unsigned *remap)
{
    const ll n = ctl->n;
    const ll base = blk * NBG_SCAN_TILE;
    if (base >= n) return;
    /* rows of NBG_SCAN_BLOCK consecutive bodies, so every field access of a
     * warp is coalesced; kept bodies keep their order */
    ll rank = blk_off[blk];
    for (int q = 0; q < NBG_SCAN_ITEMS; q++) {
        const ll k = base + (ll)q * NBG_SCAN_BLOCK + threadIdx.x;
        const bool keep = k < n && (A.flags[k] & NBG_F_EXISTS);
        ll tot;
        const ll ex = block_excl_scan(keep ? 1 : 0, &tot);
        if (keep) {
            const int sim = nbg_sim_of(seg.off, seg.nsims, k);
            const ll d = seg.new_off[sim] + (rank + ex - seg.keep_start[sim]);
            copy_body(A, k, Bt, d);
            if (remap) remap[k] = (unsigned)d;
        } else if (remap && k < n) {
            remap[k] = NBG_GONE;
        }
        rank += tot;
    }
}

__global__ void __launch_bounds__(NBG_SCAN_BLOCK) k_compact(BodyArrays A, BodyArrays Bt, DevCtl *ctl, SimSegs seg,
                                                            const ll *blk_off, unsigned *remap)
{
    if (ctl->error || !cycle_changes(ctl)) return;
    compact(A, Bt, ctl, seg, blockIdx.x, blk_off, remap);
}

/* The mixed path's Hilbert order carried through compaction: the kept bodies
 * keep their sorted sequence under their new indices, and each sim's arrivals
 * (fragments, host adds) follow its kept bodies.  A sim's sorted positions
 * cover the same range as its indices, so the stable compaction over
 * positions uses the per-sim offsets of the body compaction.  Three steps:
 * kept positions per block and, by the last block, their offsets
 * (scan_blocks mode 2), the scatter into the scratch order, and its
 * installation (order_copy). */
__device__ static void order_blocksum(const DevCtl *ctl, const unsigned *perm, const unsigned *remap, ll blk,
                                      ll *blk_sum)
{
    const ll n = ctl->n;
    const ll base = blk * NBG_SCAN_TILE;
    if (base >= n) return;
    ll s = 0;
    for (int q = 0; q < NBG_SCAN_ITEMS; q++) {
        const ll p = base + (ll)q * NBG_SCAN_BLOCK + threadIdx.x;
        s += p < n && remap[perm[p]] != NBG_GONE ? 1 : 0;
    }
    ll tot;
    block_excl_scan(s, &tot);
    if (threadIdx.x == 0) blk_sum[blk] = tot;
}

__device__ static void order_carry(const DevCtl *ctl, const SimSegs &seg, const unsigned *perm, const unsigned *remap,
                                   ll blk, const ll *blk_off, unsigned *order)
{
    const ll n = ctl->n;
    const ll base = blk * NBG_SCAN_TILE;
    if (base >= n) return;
    ll rank = blk_off[blk];
    for (int q = 0; q < NBG_SCAN_ITEMS; q++) {
        const ll p = base + (ll)q * NBG_SCAN_BLOCK + threadIdx.x;
        const unsigned to = p < n ? remap[perm[p]] : NBG_GONE;
        const bool keep = to != NBG_GONE;
        ll tot;
        const ll ex = block_excl_scan(keep ? 1 : 0, &tot);
        if (keep) {
            const int sim = nbg_sim_of(seg.off, seg.nsims, p);
            order[seg.new_off[sim] + (rank + ex - seg.keep_start[sim])] = to;
        }
        rank += tot;
    }
}

/* thread t of nt */
__device__ static void order_copy(DevCtl *ctl, const SimSegs &seg, const unsigned *order, unsigned *perm, ll t, ll nt)
{
    const ll total = seg.new_off[seg.nsims];
    for (ll k = t; k < total; k += nt) {
        const int sim = nbg_sim_of(seg.new_off, seg.nsims, k);
        perm[k] = k - seg.new_off[sim] < seg.keep[sim] ? order[k] : (unsigned)k; /* arrivals: as they come */
    }
    if (t == 0) ctl->order_carried = 1;
}

__global__ void __launch_bounds__(NBG_SCAN_BLOCK) k_order_count(DevCtl *ctl, SimSegs seg, const unsigned *perm,
                                                                const unsigned *remap, ll *blk_sum, ll *blk_off)
{
    if (ctl->error || !cycle_changes(ctl)) return;
    order_blocksum(ctl, perm, remap, blockIdx.x, blk_sum);
    if (last_block(ctl)) scan_blocks(ctl, seg, blk_sum, blk_off, 2, 0, 0);
}

__global__ void __launch_bounds__(NBG_SCAN_BLOCK) k_order_carry(DevCtl *ctl, SimSegs seg, const unsigned *perm,
                                                                const unsigned *remap, const ll *blk_off,
                                                                unsigned *order)
{
    if (ctl->error || !cycle_changes(ctl)) return;
    order_carry(ctl, seg, perm, remap, blockIdx.x, blk_off, order);
}

__global__ void k_order_copy(DevCtl *ctl, SimSegs seg, const unsigned *order, unsigned *perm)
{
    if (ctl->error || !cycle_changes(ctl)) return;
    order_copy(ctl, seg, order, perm, (ll)blockIdx.x * blockDim.x + threadIdx.x, (ll)gridDim.x * blockDim.x);
}

/* Appends each sim's adds after its kept bodies, newest first (the sim's
 * fragments of this cycle, then its host adds), each with r = R. */
__device__ static void append_adds(const BodyArrays &Bt, const BodyArrays &F, const BodyArrays &H, const DevCtl *ctl,
                                   const SimSegs &seg, ll t, ll nt)
{
    const ll nf = ctl->frag_total, nh = ctl->n_host_adds;
    const double R = ctl->R;
    const int ns = seg.nsims;
    for (ll k = t; k < nf + nh; k += nt) {
        ll d;
        if (k < nf) {
            const int s = nbg_sim_of(seg.frag_start, ns, k);
            d = seg.new_off[s] + seg.keep[s] + (seg.frag_start[s + 1] - 1 - k);
            copy_body(F, k, Bt, d);
        } else {
            const ll h = k - nf;
            const int s = nbg_sim_of(seg.hadd_start, ns, h);
            d = seg.new_off[s] + seg.keep[s] + seg.frag[s] + (seg.hadd_start[s + 1] - 1 - h);
            copy_body(H, h, Bt, d);
        }
        Bt.rest[d] = R;
    }
}

__global__ void k_append_adds(BodyArrays Bt, BodyArrays F, BodyArrays H, DevCtl *ctl, SimSegs seg)
{
    if (ctl->error || !cycle_changes(ctl)) return;
    append_adds(Bt, F, H, ctl, seg, (ll)blockIdx.x * blockDim.x + threadIdx.x, (ll)gridDim.x * blockDim.x);
}

__global__ void k_copy_back(BodyArrays A, BodyArrays Bt, DevCtl *ctl, SimSegs seg)
{
    if (ctl->error || !cycle_changes(ctl)) return;
    const ll total = seg.new_off[seg.nsims];
    for (ll k = (ll)blockIdx.x * blockDim.x + threadIdx.x; k < total; k += (ll)gridDim.x * blockDim.x)
        copy_body(Bt, k, A, k);
}

__device__ static void end_cycle(DevCtl *ctl, const SimSegs &seg)
{
    const int ns = seg.nsims;
    const bool changed = cycle_changes(ctl);
    for (int s = threadIdx.x; s <= ns; s += NBG_SCAN_BLOCK) {
        if (changed) seg.off[s] = seg.new_off[s];
        if (s < ns) seg.hadd[s] = 0;
    }
    __syncthreads(); /* every thread has read the control block */
    if (threadIdx.x != 0) return;
    const ll n = ctl->n;
    ctl->rend_n = n;
    ctl->acc_removed += n - ctl->n_keep;
    ctl->acc_interactions += ctl->cycle_interactions;
    ctl->n = ctl->n_keep + ctl->frag_total + ctl->n_host_adds;
    ctl->n_host_adds = 0;
    /* bodies changed index: the order is stale unless it was carried along */
    if (changed && !ctl->order_carried) ctl->sort_valid = 0;
    ctl->order_carried = 0;
    ctl->cycle += 1;
    ctl->acc_steps += 1;
}

__global__ void __launch_bounds__(NBG_SCAN_BLOCK) k_end(DevCtl *ctl, SimSegs seg)
{
    if (ctl->error) return;
    end_cycle(ctl, seg);
}

/* Cycle for a collection of one scan tile's capacity, by one block: kept
 * bodies, compaction, adds, the carried order (remap set) and the cycle's
 * end.  Nothing moves in most cycles: 9.6 us in place of ten launches of 29. */
__global__ void __launch_bounds__(NBG_SCAN_BLOCK) k_cycle_small(BodyArrays A, BodyArrays Bt, BodyArrays F, BodyArrays H,
                                                                DevCtl *ctl, SimSegs seg, ll *blk_sum, ll *blk_off,
                                                                unsigned *perm, unsigned *remap, unsigned *order)
{
    if (ctl->error) return;
    keep_blocksum(A, ctl, seg, 0, blk_sum);
    __syncthreads();
    scan_blocks(ctl, seg, blk_sum, blk_off, 1, 0, 0);
    if (cycle_changes(ctl)) {
        compact(A, Bt, ctl, seg, 0, blk_off, remap);
        append_adds(Bt, F, H, ctl, seg, threadIdx.x, NBG_SCAN_BLOCK);
        __syncthreads();
        const ll total = seg.new_off[seg.nsims];
        for (ll k = threadIdx.x; k < total; k += NBG_SCAN_BLOCK) copy_body(Bt, k, A, k);
        if (remap) {
            order_blocksum(ctl, perm, remap, 0, blk_sum);
            __syncthreads();
            scan_blocks(ctl, seg, blk_sum, blk_off, 2, 0, 0);
            order_carry(ctl, seg, perm, remap, 0, blk_off, order);
            __syncthreads();
            order_copy(ctl, seg, order, perm, threadIdx.x, NBG_SCAN_BLOCK);
        }
        __syncthreads();
    }
    end_cycle(ctl, seg);
}

/* ------------------------------------------------------------------------ */
/* cycle-boundary edits                                                     */
/* ------------------------------------------------------------------------ */

/* Bodies [lo, hi) of collection sim (sim < 0: the whole array). */
__device__ __forceinline__ void sim_range(const DevCtl *ctl, const SimSegs &seg, int sim, ll &lo, ll &hi)
{
    lo = sim >= 0 ? seg.off[sim] : 0;
    hi = sim >= 0 ? seg.off[sim + 1] : ctl->n;
}

/* processDeletes, computation-runner.go:176-216 (sequential by nature), over
 * collection sim (sim < 0: the whole array, one collection). */
__global__ void k_remove(BodyArrays A, DevCtl *ctl, SimSegs seg, int sim, ll count, ll *removed)
{
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    ll lo, hi;
    sim_range(ctl, seg, sim, lo, hi);
    const ll n = hi - lo;
    ll rem = 0;
    if (count == -1) {
        for (ll k = lo; k < hi; k++) {
            if (A.flags[k] & NBG_F_EXISTS) {
                A.m[k] = 0;
                A.flags[k] &= ~NBG_F_EXISTS;
                rem++;
            }
        }
    } else if (n > 0) {
        const ll step = count > n ? 1 : n / count;
        ll iter = 0;
        bool should = false;
        for (ll k = lo; k < hi; k++) {
            if (iter % step == 0) should = true;
            iter++;
            unsigned f = A.flags[k];
            if (should && !(f & NBG_F_PINNED) && (f & NBG_F_EXISTS)) {
                A.m[k] = 0;
                A.flags[k] = f & ~NBG_F_EXISTS;
                should = false;
                rem++;
            }
        }
    }
    *removed = rem;
}

/* ApplyMods for bodies matched by id (body.go:274-313, after parsing), in
 * collection sim (sim < 0: every collection). */
__global__ void k_edits(BodyArrays A, DevCtl *ctl, SimSegs seg, int sim, const nbg_edit *E, ll ne, int *results)
{
    ll lo, hi;
    sim_range(ctl, seg, sim, lo, hi);
    for (ll k = lo + (ll)blockIdx.x * blockDim.x + threadIdx.x; k < hi; k += (ll)gridDim.x * blockDim.x) {
        const ll id = A.id[k];
        for (ll q = 0; q < ne; q++) {
            const nbg_edit e = E[q];
            if (e.id != id) continue;
            atomicAdd(&results[q], 1);
            const unsigned m = e.mask;
            if (m & NBG_M_X) A.x[k] = e.x;
            if (m & NBG_M_Y) A.y[k] = e.y;
            if (m & NBG_M_Z) A.z[k] = e.z;
            if (m & NBG_M_VX) A.vx[k] = e.vx;
            if (m & NBG_M_VY) A.vy[k] = e.vy;
            if (m & NBG_M_VZ) A.vz[k] = e.vz;
            if (m & NBG_M_MASS) A.m[k] = e.mass;
            if (m & NBG_M_RADIUS) A.rad[k] = e.radius;
            if (m & NBG_M_FRAG_FACTOR) A.ff[k] = e.frag_factor;
            if (m & NBG_M_FRAG_STEP) A.fs[k] = e.frag_step;
            unsigned f = A.flags[k];
            if (m & NBG_M_COLLISION)
                f = (f & ~(3u << NBG_BEHAVIOR_SHIFT)) | (((unsigned)e.collision & 3u) << NBG_BEHAVIOR_SHIFT);
            if (m & NBG_M_TELEMETRY) f = e.telemetry ? (f | NBG_F_TELEMETRY) : (f & ~NBG_F_TELEMETRY);
            if (m & NBG_M_EXISTS) f = e.exists ? (f | NBG_F_EXISTS) : (f & ~NBG_F_EXISTS);
            A.flags[k] = f;
        }
    }
}

/* The first body with this id in collection sim (sim < 0: anywhere). */
__global__ void k_find(BodyArrays A, DevCtl *ctl, SimSegs seg, int sim, ll id, ll *idx)
{
    ll lo, hi;
    sim_range(ctl, seg, sim, lo, hi);
    for (ll k = lo + (ll)blockIdx.x * blockDim.x + threadIdx.x; k < hi; k += (ll)gridDim.x * blockDim.x)
        if (A.id[k] == id) atomicMin((long long *)idx, (long long)k);
}

/* dst[k] = src[index[k]] for k < n: every field of a body record. */
__global__ void k_gather_bodies(BodyArrays S, BodyArrays D, const ll *index, ll n)
{
    for (ll k = (ll)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += (ll)gridDim.x * blockDim.x)
        copy_body(S, index[k], D, k);
}

/* Kinetic and pairwise potential energy plus momentum, per-block partials
 * (out[blockIdx*5 + 0..4]) summed on the host in block order. */
#define EN_BLOCK 128
__global__ void __launch_bounds__(EN_BLOCK) k_energy(BodyArrays A, DevCtl *ctl, SimSegs seg, double *out)
{
    __shared__ double red[5][EN_BLOCK];
    const ll n = ctl->n;
    double ke = 0, pe = 0, px = 0, py = 0, pz = 0;
    const ll i = (ll)blockIdx.x * EN_BLOCK + threadIdx.x;
    if (i < n && (A.flags[i] & NBG_F_EXISTS)) {
        const double m = A.m[i], vx = A.vx[i], vy = A.vy[i], vz = A.vz[i];
        ke = 0.5 * m * (vx * vx + vy * vy + vz * vz);
        px = m * vx;
        py = m * vy;
        pz = m * vz;
        const double xi = A.x[i], yi = A.y[i], zi = A.z[i];
        const ll end = seg.off[nbg_sim_of(seg.off, seg.nsims, i) + 1]; /* pairs within i's sim */
        for (ll j = i + 1; j < end; j++) {
            if (!(A.flags[j] & NBG_F_EXISTS)) continue;
            const double dx = A.x[j] - xi, dy = A.y[j] - yi, dz = A.z[j] - zi;
            const double r = sqrt(dx * dx + dy * dy + dz * dz);
            if (r > 0) pe -= NBG_G * m * A.m[j] / r;
        }
    }
    red[0][threadIdx.x] = ke;
    red[1][threadIdx.x] = pe;
    red[2][threadIdx.x] = px;
    red[3][threadIdx.x] = py;
    red[4][threadIdx.x] = pz;
    __syncthreads();
    for (int s = EN_BLOCK / 2; s > 0; s >>= 1) {
        if (threadIdx.x < s)
            for (int q = 0; q < 5; q++) red[q][threadIdx.x] += red[q][threadIdx.x + s];
        __syncthreads();
    }
    if (threadIdx.x == 0)
        for (int q = 0; q < 5; q++) out[(ll)blockIdx.x * 5 + q] = red[q][0];
}

/* ------------------------------------------------------------------------ */
/* launchers                                                                */
/* ------------------------------------------------------------------------ */

static int scan_grid(ll cap) { return (int)((cap + NBG_SCAN_TILE - 1) / NBG_SCAN_TILE); }


/* whether one block of each cycle kernel covers the collections */
static bool small_cycle(const CycleBufs &cb) { return cb.cap <= NBG_SCAN_TILE; }

/* direct: the mixed direct sum follows, whose symmetric kernel needs its j
 * partials; no other force pass reads them, whatever the shape */
void nbg_launch_begin(const CycleBufs &cb, DevCtl *ctl, cudaStream_t st, bool direct)
{
    k_begin<<<1, NBG_SCAN_BLOCK, 0, st>>>(ctl, cb.seg, cb.slots, cb.work_cap, cb.itile > 0 ? cb.itile : NBG_MIX_ITILE,
                                          cb.part_doubles, direct && nbg_mix_is_sym(cb.mix_variant), cb.jpart_units);
}

void nbg_launch_begin_cycle(const CycleBufs &cb, DevCtl *ctl, cudaStream_t st, bool direct)
{
    if (small_cycle(cb)) {
        k_begin_small<<<1, NBG_SCAN_BLOCK, 0, st>>>(
            cb.a, ctl, cb.seg, cb.slots, cb.work_cap, cb.itile > 0 ? cb.itile : NBG_MIX_ITILE, cb.part_doubles,
            direct && nbg_mix_is_sym(cb.mix_variant), cb.jpart_units, cb.blk_sum, cb.blk_off, cb.cap, cb.frag_cap);
        return;
    }
    nbg_launch_begin(cb, ctl, st, direct);
    k_frag_count<<<scan_grid(cb.cap), NBG_SCAN_BLOCK, 0, st>>>(cb.a, ctl, cb.seg, cb.blk_sum, cb.blk_off, cb.cap,
                                                               cb.frag_cap);
}

void nbg_launch_pair_fp64(const CycleBufs &cb, DevCtl *ctl, cudaStream_t st)
{
    /* one wave of resident CTAs, which take blocks of bodies from a counter */
    const ll sms = cb.sms > 0 ? cb.sms : 1;
    const ll most = (cb.cap + 3) / 4 + cb.seg.nsims;
    auto *const k = cb.seg.nsims > 1 ? k_pair_fp64<true> : k_pair_fp64<false>;
    cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(P64Shared));
    k<<<(unsigned)(most < P64_MINB * sms ? most : P64_MINB * sms), P64_THREADS, sizeof(P64Shared), st>>>(
        cb.a, ctl, cb.seg, cb.ev_keys, cb.ev_cap);
}

/* everything after the pair kernel: order events, emit fragments, resolve,
 * integrate, Cycle */
void nbg_launch_after_pair(const CycleBufs &cb, DevCtl *ctl, cudaStream_t st, bool carry_order)
{
    const int sg = scan_grid(cb.cap);
    const bool small = small_cycle(cb);
    if (small && !cb.ev_radix)
        k_events_small<<<1, SORT_BLOCK, 0, st>>>(cb.a, cb.frags, ctl, cb.ev_keys, cb.ev_cap, cb.blk_off);
    else
        k_sort_events<<<1, SORT_BLOCK, 0, st>>>(ctl, cb.ev_keys, cb.ev_cap, cb.ev_radix);
    int links = 0;
    if (cb.ev_radix) {
        nbg_launch_event_radix(cb, ctl, st);
        /* the links, when a body index and an event index fit one key */
        int kb = 1, ob = 1;
        while (kb < 31 && ((ll)1 << kb) < cb.cap) kb++;
        while (ob < 40 && ((ll)1 << ob) < cb.ev_cap) ob++;
        if (kb + ob + 1 <= 64) {
            links = 1;
            const int eg = nbg_flat_grid(cb, 2 * cb.ev_cap);
            k_ev_ranges<<<(cb.seg.nsims + 256) / 256, 256, 0, st>>>(ctl, cb.seg, cb.ev_keys, cb.ev_lo);
            k_ev_incid<<<eg, 256, 0, st>>>(ctl, cb.seg, cb.ev_keys, cb.ev_lo, cb.inc[0], ob);
            const ull *sorted = nbg_launch_incidence_radix(cb, ctl, kb + ob, st);
            k_ev_links<<<eg, 256, 0, st>>>(ctl, sorted, ob, cb.ev_link, cb.ev_front);
            k_ev_pending<<<eg, 256, 0, st>>>(ctl, cb.ev_front, cb.ev_pend);
        }
    }
    if (!small || cb.ev_radix) k_frag_emit<<<sg, NBG_SCAN_BLOCK, 0, st>>>(cb.a, cb.frags, ctl, cb.blk_off);
    /* the radix-sort key buffer is free after the pair pass: per-body owner words */
    k_resolve<<<cb.seg.nsims, RESOLVE_BLOCK, 0, st>>>(cb.a, ctl, cb.seg, cb.ev_keys, cb.ev_out, cb.skey[1], links,
                                                      cb.ev_lo, cb.ev_link, cb.ev_pend, cb.ev_front, cb.ev_cap);
    k_integrate<<<nbg_flat_grid(cb, cb.cap), 256, 0, st>>>(cb.a, ctl, cb.rend, cb.ring_rend, cb.ring_cap, cb.ring_slots);
    if (cb.ring_head) k_ring_header<<<1, 1, 0, st>>>(ctl, cb.ring_head, cb.ring_cap, cb.ring_slots);
    /* the radix value buffer is free after the sort: old -> new index; the
     * sorted-key buffer too: the scratch order */
    unsigned *remap = carry_order ? cb.sval : nullptr;
    if (small) {
        k_cycle_small<<<1, NBG_SCAN_BLOCK, 0, st>>>(cb.a, cb.b, cb.frags, cb.adds, ctl, cb.seg, cb.blk_sum, cb.blk_off,
                                                    cb.perm, remap, cb.skey[0]);
        return;
    }
    k_keep_count<<<sg, NBG_SCAN_BLOCK, 0, st>>>(cb.a, ctl, cb.seg, cb.blk_sum, cb.blk_off);
    k_compact<<<sg, NBG_SCAN_BLOCK, 0, st>>>(cb.a, cb.b, ctl, cb.seg, cb.blk_off, remap);
    k_append_adds<<<nbg_flat_grid(cb, cb.frag_cap + cb.adds_cap), 256, 0, st>>>(cb.b, cb.frags, cb.adds, ctl, cb.seg);
    k_copy_back<<<nbg_flat_grid(cb, cb.cap), 256, 0, st>>>(cb.a, cb.b, ctl, cb.seg);
    if (carry_order) {
        k_order_count<<<sg, NBG_SCAN_BLOCK, 0, st>>>(ctl, cb.seg, cb.perm, remap, cb.blk_sum, cb.blk_off);
        k_order_carry<<<sg, NBG_SCAN_BLOCK, 0, st>>>(ctl, cb.seg, cb.perm, remap, cb.blk_off, cb.skey[0]);
        k_order_copy<<<nbg_flat_grid(cb, cb.cap), 256, 0, st>>>(ctl, cb.seg, cb.skey[0], cb.perm);
    }
    k_end<<<1, NBG_SCAN_BLOCK, 0, st>>>(ctl, cb.seg);
}

/* launches of nbg_launch_begin_cycle and nbg_launch_after_pair (without the
 * multi-block event sort and the render ring's header) */
int nbg_cycle_launches(const CycleBufs &cb, bool carry_order)
{
    if (small_cycle(cb)) return 1 + (cb.ev_radix ? 2 : 1) + 2 + 1;
    return 2 + 4 + 5 + (carry_order ? 3 : 0);
}

void nbg_launch_remove(const CycleBufs &cb, DevCtl *ctl, int sim, ll count, ll *removed_dev, cudaStream_t st)
{
    k_remove<<<1, 32, 0, st>>>(cb.a, ctl, cb.seg, sim, count, removed_dev);
}

void nbg_launch_edits(const CycleBufs &cb, DevCtl *ctl, int sim, const nbg_edit *edits_dev, ll k, int *results_dev,
                      cudaStream_t st)
{
    k_edits<<<nbg_flat_grid(cb, cb.cap), 256, 0, st>>>(cb.a, ctl, cb.seg, sim, edits_dev, k, results_dev);
}

void nbg_launch_find(const CycleBufs &cb, DevCtl *ctl, int sim, ll id, ll *idx_dev, cudaStream_t st)
{
    k_find<<<nbg_flat_grid(cb, cb.cap), 256, 0, st>>>(cb.a, ctl, cb.seg, sim, id, idx_dev);
}

void nbg_launch_gather(const CycleBufs &cb, const BodyArrays &src, const BodyArrays &dst, const ll *index_dev, ll n,
                       cudaStream_t st)
{
    if (n > 0) k_gather_bodies<<<nbg_flat_grid(cb, n), 256, 0, st>>>(src, dst, index_dev, n);
}

void nbg_launch_energy(const CycleBufs &cb, DevCtl *ctl, double *out_dev, cudaStream_t st)
{
    int g = (int)((cb.cap + EN_BLOCK - 1) / EN_BLOCK);
    k_energy<<<g, EN_BLOCK, 0, st>>>(cb.a, ctl, cb.seg, out_dev);
}
