/*
 * k_bh.cu - the Barnes-Hut force pass (cmd/body/octree.go) on the GPU.
 *
 * The reference builds a point-region octree by inserting the bodies that
 * exist and are not fragmenting, in array order, into a cube centred on
 * their bounding box (half = max extent / 2 * 1.05, octree.go:136-188); a
 * leaf holds one body, and an occupied leaf that receives another splits
 * into eight children.  Which node each body ends in depends only on the
 * comparisons x >= cx, y >= cy, z >= cz down the tree (octantOf,
 * octree.go:53-65), so the tree is built here without insertion:
 *
 *   1. every tree body descends BH_LEVELS levels with the reference's own
 *      centre arithmetic (cx +- half / 2, half / 2) and records its octant
 *      path, 3 bits a level, as a 63-bit key;
 *   2. the keys are sorted (LSD radix, stable);
 *   3. a node is a key prefix shared by at least one body whose parent holds
 *      two or more: the nodes that start at sorted position p run from the
 *      first level where key p differs from key p - 1 down to the level
 *      where it parts from key p + 1, so their count comes from the two
 *      neighbouring keys, and one scan numbers every node in depth-first
 *      order (position, then level).  That order makes the first child of a
 *      node the next node and the end of its subtree the first node starting
 *      at the end of its body range (the skip pointer), so the force pass
 *      walks the tree without a stack;
 *   4. masses and moments are summed from the leaves up, in one launch, over
 *      the children in octant order.
 *
 * The force pass (accumForce, octree.go:265-305) walks the tree for every
 * body with the reference's expressions, softening 1e-4 and opening angle
 * 0.3; a sun sums every body directly (CalcForce, octree.go:236-263).  The
 * collision pass (Compute's second loop, body.go:171-186) becomes a range
 * query on the same tree: nodes whose cube lies farther than r_i + r_max are
 * skipped, and every body that remains is tested with the reference's exact
 * dist <= r_i + r_j, so the event set is the O(N^2) loop's.  Bodies outside
 * the tree (not existing, fragmenting, or not finite) are tested one by one.
 *
 * Against the reference's tree:
 *  - the tree and the opening decisions are the same; a node's centre of
 *    mass is sum(m x) / sum(m) instead of the reference's running update,
 *    which differs in the last bits (a one-body leaf is x * m / m, as in the
 *    reference).  The reference's node whose first inserted body is massless
 *    has a NaN centre (0 / 0) and is therefore always opened; that is kept;
 *  - keys have 21 levels; bodies that share a node at that depth (closer
 *    than 2^-20 of the root cube) stay together in one leaf and each acts as
 *    a leaf of its own, where the reference keeps splitting (and recurses
 *    without end for two bodies at one position);
 *  - the sun's direct sum is a parallel reduction, not array order.
 *
 * Several collections (nbg_set_collections): one tree per collection, each
 * exactly the tree a context holding that collection alone builds.  Every
 * collection gets its own bounding box and root cube; after the key passes
 * the sort takes two more stable passes on the collection index (tree
 * bodies; the others go last), so each collection's tree bodies are one run
 * of sorted positions, in key order.  Node boundaries are found within each
 * run, the depth-first numbering then puts each collection's nodes in one
 * range with its root first, and the walks, the suns' sums and the collision
 * query stay inside the body's own collection.  Walk groups of 32 bodies
 * start at each collection's first sorted position, as they would alone.
 */
#include "nbg_exact.h"
#include "nbg_internal.cuh"
#include "nbg_math.h"
#include "nbg_octant.h"
#include "nbg_radix.cuh"
#include "nbg_shared.h"

#define BH_THETA 0.3
#define BH_FLT_MAX 3.402823466e38f
#define BH_SOFTENING 1e-4
#define BH_LEVELS NBG_OCT_LEVELS
#define BH_BLOCK 256
#define BH_RS_PASSES 10
#define BH_SCAN_BLOCK 1024
#define BH_SCAN_ITEMS 4
#define BH_SCAN_TILE (BH_SCAN_BLOCK * BH_SCAN_ITEMS)
#define BHW_BLOCK 128 /* the mixed walk's CTAs */
#define BHW_TEAM (BHW_BLOCK / 32)
/* Collections of at least this many tree bodies have a warp to each group of
 * 32 bodies; in smaller ones, whose groups would leave warps idle, a CTA's
 * four warps share a group's walk.  Tree pass, a warp to a group against four:
 * 30,011 Plummer bodies 1.33 / 1.07 ms, 131,072 2.38 / 2.89 ms, 400,000
 * 5.8 / 7.5 ms (the four repeat the top of the tree).  Decided for each
 * collection by its own size, so its sums are those it has alone. */
#ifndef BHW_SOLO_MIN
#define BHW_SOLO_MIN 60000
#endif
#define BH_F_LEAF 1u
#define BH_F_NAN_CM 2u
#define BH_F_FAR_OUT 8u /* mixed walk: a one-body leaf past FP32's range */
#define FULL_MASK 0xffffffffu

/* order-preserving integer image of a double (for atomicMin / atomicMax) */
__device__ __forceinline__ ull dbl_ord(double v)
{
    const ull b = (ull)__double_as_longlong(v);
    return (b >> 63) ? ~b : (b | 0x8000000000000000ull);
}
__device__ __forceinline__ double ord_dbl(ull o)
{
    const ull b = (o >> 63) ? (o & 0x7fffffffffffffffull) : ~o;
    return __longlong_as_double((long long)b);
}

__device__ __forceinline__ bool tree_body(const BodyArrays &A, ll k)
{
    if ((A.flags[k] & NBG_LIVE_MASK) != NBG_F_EXISTS) return false;
    const double x = A.x[k], y = A.y[k], z = A.z[k];
    return fabs(x) <= NBG_DBL_MAX && fabs(y) <= NBG_DBL_MAX && fabs(z) <= NBG_DBL_MAX;
}

/* the root cube of collection s, octree.go:174-183 */
__device__ __forceinline__ void bh_root(const BhTree &t, int s, double &cx, double &cy, double &cz, double &half)
{
    const ull *b = t.sbox + 6 * (ll)s;
    const double minX = ord_dbl(b[0]), minY = ord_dbl(b[1]), minZ = ord_dbl(b[2]);
    const double maxX = ord_dbl(b[3]), maxY = ord_dbl(b[4]), maxZ = ord_dbl(b[5]);
    cx = (minX + maxX) / 2;
    cy = (minY + maxY) / 2;
    cz = (minZ + maxZ) / 2;
    half = nbg_go_max(maxX - minX, nbg_go_max(maxY - minY, maxZ - minZ)) / 2 * 1.05;
}

/* ---- 1. bounds, keys -------------------------------------------------------- */

/* empty boxes and counts for every collection, and no digits counted */
__global__ void __launch_bounds__(1024) k_bh_reset(DevCtl *ctl, SimSegs seg, BhTree t)
{
    if (ctl->error) return;
    for (int d = threadIdx.x; d < BH_RS_PASSES * RX_BINS; d += blockDim.x) t.digits[d] = 0;
    for (int s = threadIdx.x; s < seg.nsims; s += blockDim.x) {
        ull *b = t.sbox + 6 * (ll)s;
        for (int c = 0; c < 3; c++) {
            b[c] = ~0ull;
            b[3 + c] = 0ull;
        }
        t.scount[s] = 0;
    }
}

/* each collection's bounding box and tree-body count, and the largest
 * radius of any body */
__global__ void __launch_bounds__(BH_BLOCK) k_bh_bounds(BodyArrays A, DevCtl *ctl, SimSegs seg, BhTree t)
{
    if (ctl->error) return;
    const ll n = ctl->n;
    const int lane = threadIdx.x & 31;
    double rmax = 0;
    ull lo[3] = {~0ull, ~0ull, ~0ull}, hi[3] = {0ull, 0ull, 0ull};
    unsigned cnt = 0;
    if (seg.nsims == 1) {
        /* one collection: a lane keeps its own box, and the warp reduces once
         * (reducing every 32 bodies, as below, took 83 us for 1,048,576 against
         * 34) */
        for (ll k = (ll)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += (ll)gridDim.x * blockDim.x) {
            const double r = A.rad[k];
            if (r > rmax) rmax = r;
            if (!tree_body(A, k)) continue;
            const ull p[3] = {dbl_ord(A.x[k]), dbl_ord(A.y[k]), dbl_ord(A.z[k])};
            for (int c = 0; c < 3; c++) {
                lo[c] = p[c] < lo[c] ? p[c] : lo[c];
                hi[c] = p[c] > hi[c] ? p[c] : hi[c];
            }
            cnt++;
        }
        for (int o = 16; o > 0; o >>= 1) {
            for (int c = 0; c < 3; c++) {
                const ull l = __shfl_xor_sync(FULL_MASK, lo[c], o), h = __shfl_xor_sync(FULL_MASK, hi[c], o);
                lo[c] = l < lo[c] ? l : lo[c];
                hi[c] = h > hi[c] ? h : hi[c];
            }
            cnt += __shfl_xor_sync(FULL_MASK, cnt, o);
        }
        if (lane == 0 && cnt > 0) {
            for (int c = 0; c < 3; c++) {
                atomicMin((unsigned long long *)&t.sbox[c], (unsigned long long)lo[c]);
                atomicMax((unsigned long long *)&t.sbox[3 + c], (unsigned long long)hi[c]);
            }
            atomicAdd((unsigned long long *)&t.scount[0], (unsigned long long)cnt);
        }
    } else
    /* warp-uniform trip count: every lane takes part in the reductions */
    for (ll base = (ll)blockIdx.x * blockDim.x; base < n; base += (ll)gridDim.x * blockDim.x) {
        const ll k = base + threadIdx.x;
        for (int c = 0; c < 3; c++) {
            lo[c] = ~0ull;
            hi[c] = 0ull;
        }
        cnt = 0;
        int sim = -1;
        if (k < n) {
            const double r = A.rad[k];
            if (r > rmax) rmax = r;
            sim = nbg_sim_of(seg.off, seg.nsims, k);
            if (tree_body(A, k)) {
                lo[0] = hi[0] = dbl_ord(A.x[k]);
                lo[1] = hi[1] = dbl_ord(A.y[k]);
                lo[2] = hi[2] = dbl_ord(A.z[k]);
                cnt = 1;
            }
        }
        /* bodies lie in collection order, so the collections of a warp are
         * runs of lanes: a segmented reduction down each run leaves its sum
         * in the run's first lane */
        for (int o = 1; o < 32; o <<= 1) {
            const int so = __shfl_down_sync(FULL_MASK, sim, o);
            ull l[3], h[3];
            for (int c = 0; c < 3; c++) {
                l[c] = __shfl_down_sync(FULL_MASK, lo[c], o);
                h[c] = __shfl_down_sync(FULL_MASK, hi[c], o);
            }
            const unsigned co = __shfl_down_sync(FULL_MASK, cnt, o);
            if (lane + o < 32 && so == sim) {
                for (int c = 0; c < 3; c++) {
                    lo[c] = l[c] < lo[c] ? l[c] : lo[c];
                    hi[c] = h[c] > hi[c] ? h[c] : hi[c];
                }
                cnt += co;
            }
        }
        const int sprev = __shfl_up_sync(FULL_MASK, sim, 1);
        if (sim >= 0 && cnt > 0 && (lane == 0 || sprev != sim)) {
            ull *b = t.sbox + 6 * (ll)sim;
            for (int c = 0; c < 3; c++) {
                atomicMin((unsigned long long *)&b[c], (unsigned long long)lo[c]);
                atomicMax((unsigned long long *)&b[3 + c], (unsigned long long)hi[c]);
            }
            atomicAdd((unsigned long long *)&t.scount[sim], (unsigned long long)cnt);
        }
    }
    for (int o = 16; o > 0; o >>= 1) rmax = fmax(rmax, __shfl_xor_sync(FULL_MASK, rmax, o));
    if (lane == 0) atomicMax((unsigned long long *)&ctl->bh_rmax, (unsigned long long)dbl_ord(rmax));
}

/* each collection's first sorted position and first walk group (exclusive
 * scans over the collections, one warp), and the tree-body total */
__global__ void __launch_bounds__(32) k_bh_segs(DevCtl *ctl, SimSegs seg, BhTree t)
{
    if (ctl->error) return;
    const int ns = seg.nsims, lane = threadIdx.x;
    const int per = (ns + 31) / 32;
    const int s0 = lane * per, s1 = s0 + per < ns ? s0 + per : ns;
    /* units of the mixed walk: a group, or a CTA's warps' worth of them */
    auto units = [&](int s) {
        const ll gr = (t.scount[s] + 31) / 32;
        return t.scount[s] >= BHW_SOLO_MIN ? (gr + BHW_TEAM - 1) / BHW_TEAM : gr;
    };
    ll c = 0, g = 0, u = 0;
    for (int s = s0; s < s1; s++) {
        c += t.scount[s];
        g += (t.scount[s] + 31) / 32;
        u += units(s);
    }
    ll xc = c, xg = g, xu = u;
    for (int o = 1; o < 32; o <<= 1) {
        const ll yc = __shfl_up_sync(FULL_MASK, xc, o), yg = __shfl_up_sync(FULL_MASK, xg, o);
        const ll yu = __shfl_up_sync(FULL_MASK, xu, o);
        if (lane >= o) {
            xc += yc;
            xg += yg;
            xu += yu;
        }
    }
    ll oc = xc - c, og = xg - g, ou = xu - u;
    for (int s = s0; s < s1; s++) {
        t.stree[s] = oc;
        t.sgrp[s] = og;
        t.sunit[s] = ou;
        oc += t.scount[s];
        og += (t.scount[s] + 31) / 32;
        ou += units(s);
    }
    if (lane == 31) {
        t.stree[ns] = xc;
        t.sgrp[ns] = xg;
        t.sunit[ns] = xu;
        ctl->bh_count = xc;
    }
}

/* the collection whose run of sorted tree positions holds p (0 <= p < M) */
__device__ __forceinline__ int bh_run_of(const BhTree &t, int nsims, ll p) { return nbg_sim_of(t.stree, nsims, p); }

/* a collection's root cube as a grid */
__device__ __forceinline__ NbgOctGrid bh_grid(const BhTree &t, int s)
{
    double cx, cy, cz, half;
    bh_root(t, s, cx, cy, cz, half);
    return nbg_oct_grid(cx, cy, cz, half);
}

/* the path of the rare body near a cell's face */
__device__ __noinline__ ull bh_path(double x, double y, double z, double cx, double cy, double cz, double half)
{
    return nbg_oct_path(x, y, z, cx, cy, cz, half);
}

/* Octant path of every tree body in its collection's cube; other bodies get the
 * largest key.  The 21 levels' comparisons and centres are 170 FP64 operations a
 * body, and the FP64 pipe bounds the pass; the cell of a 2^21 grid has the same bits unless the
 * coordinate is within rounding of a cell's face, which takes 9 (and the path
 * where it is): 49 -> 18 us at 131,072 bodies, 252 -> 38 us at 1,048,576. */
__global__ void __launch_bounds__(BH_BLOCK) k_bh_keys(BodyArrays A, DevCtl *ctl, SimSegs seg, BhTree t, ull *keys,
                                                      unsigned *vals)
{
    if (ctl->error) return;
    const ll n = ctl->n;
    int sim = -1;
    NbgOctGrid g;
    for (ll k = (ll)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += (ll)gridDim.x * blockDim.x) {
        ull key = ~0ull;
        if (tree_body(A, k)) {
            const double x = A.x[k], y = A.y[k], z = A.z[k];
            const int s = nbg_sim_of(seg.off, seg.nsims, k);
            if (s != sim) {
                g = bh_grid(t, s);
                sim = s;
            }
            if (!nbg_oct_cell(g, x, y, z, key)) key = bh_path(x, y, z, g.cx, g.cy, g.cz, g.half);
        }
        keys[k] = key;
        vals[k] = (unsigned)k;
    }
}

/* ---- 2. 64-bit LSD radix sort (stable) ----------------------------------- */

/* The digit of a sort pass: 8 bits of the key (simpass < 0), or, in the
 * two passes that group the tree bodies by collection, 8 bits of the
 * collection index (nsims for a body outside the trees, so those go last) */
__device__ __forceinline__ unsigned bh_digit(const SimSegs &seg, ull key, unsigned val, int shift, int simpass)
{
    if (simpass < 0) return (unsigned)(key >> shift) & 0xffu;
    const unsigned d = key == ~0ull ? (unsigned)seg.nsims : (unsigned)nbg_sim_of(seg.off, seg.nsims, (ll)val);
    return (d >> (8 * simpass)) & 0xffu;
}

/* (nbg_radix.cuh; a pass over 131,072 keys takes 12.6 us with the scan, 30.9 with
 * tiles of 4,096 and a scan by one block, over 1,048,576 28.6 and 63.8) */
__global__ void __launch_bounds__(RX_BLOCK) k_bh_rs_hist(DevCtl *ctl, SimSegs seg, const ull *keys,
                                                       const unsigned *vals, int shift, int simpass, int wide,
                                                       unsigned *hist, unsigned *digits)
{
    if (ctl->error) return;
    rx_hist(ctl->n, wide, hist, digits,
            [&](ll k) { return bh_digit(seg, keys[k], simpass < 0 ? 0u : vals[k], shift, simpass); });
}

__global__ void __launch_bounds__(RX_BLOCK) k_bh_rs_scan(DevCtl *ctl, unsigned *hist, const unsigned *digits)
{
    if (ctl->error) return;
    rx_scan(ctl->n, hist, digits);
}

__global__ void __launch_bounds__(RX_BLOCK) k_bh_rs_scatter(DevCtl *ctl, SimSegs seg, const ull *keys_in,
                                                          const unsigned *vals_in, ull *keys_out, unsigned *vals_out,
                                                          int shift, int simpass, int wide, const unsigned *hist,
                                                          const unsigned *digits)
{
    if (ctl->error) return;
    rx_scatter(ctl->n, wide, keys_in, vals_in, keys_out, vals_out, hist, digits,
               [&](ull key, unsigned val) { return bh_digit(seg, key, val, shift, simpass); });
}

/* ---- 3. nodes -------------------------------------------------------------- */

/* levels two keys have in common (BH_LEVELS when equal) */
__device__ __forceinline__ int common_levels(ull a, ull b)
{
    const ull x = a ^ b;
    if (x == 0) return BH_LEVELS;
    return (__clzll((long long)x) - 1) / 3;
}

/* first and last level of the nodes that start at sorted position p of its
 * collection's run [lo, hi) (none when first > last) */
__device__ __forceinline__ void node_levels(const ull *keys, ll p, ll lo, ll hi, int &d0, int &d1)
{
    const int cp = p == lo ? -1 : common_levels(keys[p - 1], keys[p]);
    const int cn = p == hi - 1 ? -1 : common_levels(keys[p], keys[p + 1]);
    d0 = p == lo ? 0 : cp + 1;
    const int e = cn + 1 > d0 ? cn + 1 : d0;
    d1 = e < BH_LEVELS ? e : BH_LEVELS;
}

/* per-block sums of the node counts of sorted positions [0, M) */
__global__ void __launch_bounds__(BH_SCAN_BLOCK) k_bh_count(DevCtl *ctl, SimSegs seg, BhTree t, const ull *keys,
                                                            ll *base, ll *blk)
{
    __shared__ ll red[BH_SCAN_BLOCK / 32];
    if (ctl->error) return;
    const ll M = ctl->bh_count;
    const ll b0 = (ll)blockIdx.x * BH_SCAN_TILE;
    if (b0 > M) return;
    ll s = 0;
    for (int q = 0; q < BH_SCAN_ITEMS; q++) {
        const ll p = b0 + (ll)q * BH_SCAN_BLOCK + threadIdx.x;
        ll c = 0;
        if (p < M) {
            const int r = bh_run_of(t, seg.nsims, p);
            int d0, d1;
            node_levels(keys, p, t.stree[r], t.stree[r + 1], d0, d1);
            c = d1 >= d0 ? d1 - d0 + 1 : 0;
        }
        if (p <= M) base[p] = c; /* base[M] = 0: the scan leaves the total there */
        s += c;
    }
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(FULL_MASK, s, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        ll t = 0;
        for (int w = 0; w < BH_SCAN_BLOCK / 32; w++) t += red[w];
        blk[blockIdx.x] = t;
    }
}

/* exclusive scan of the block sums (one block) and the node total */
__global__ void __launch_bounds__(1024) k_bh_count_top(DevCtl *ctl, ll *blk, ll node_cap)
{
    __shared__ ll warp_tot[32];
    if (ctl->error) return;
    const ll M = ctl->bh_count;
    const ll nblk = M / BH_SCAN_TILE + 1;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    ll carry = 0;
    for (ll c0 = 0; c0 < nblk; c0 += 1024) {
        const ll c = c0 + threadIdx.x;
        const ll v = c < nblk ? blk[c] : 0;
        ll x = v;
        for (int o = 1; o < 32; o <<= 1) {
            const ll y = __shfl_up_sync(FULL_MASK, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) warp_tot[w] = x;
        __syncthreads();
        if (w == 0) {
            ll t = warp_tot[lane];
            for (int o = 1; o < 32; o <<= 1) {
                const ll y = __shfl_up_sync(FULL_MASK, t, o);
                if (lane >= o) t += y;
            }
            warp_tot[lane] = t;
        }
        __syncthreads();
        if (c < nblk) blk[c] = carry + x - v + (w > 0 ? warp_tot[w - 1] : 0);
        carry += warp_tot[31];
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        ctl->bh_nodes = carry;
        if (carry > node_cap) {
            ctl->error = NBG_E_OVERFLOW;
            ctl->error_what = 5;
            ctl->error_need = carry;
        }
    }
}

/* exclusive scan of the node counts within each block, plus the block's
 * offset: base[p] = first node starting at p, base[M] = node total */
__global__ void __launch_bounds__(BH_SCAN_BLOCK) k_bh_count_scan(DevCtl *ctl, ll *base, const ll *blk)
{
    __shared__ ll warp_tot[32];
    if (ctl->error) return;
    const ll M = ctl->bh_count;
    const ll b0 = (ll)blockIdx.x * BH_SCAN_TILE;
    if (b0 > M) return;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    ll carry = blk[blockIdx.x];
    for (int q = 0; q < BH_SCAN_ITEMS; q++) {
        const ll p = b0 + (ll)q * BH_SCAN_BLOCK + threadIdx.x;
        const ll v = p <= M ? base[p] : 0;
        ll x = v;
        for (int o = 1; o < 32; o <<= 1) {
            const ll y = __shfl_up_sync(FULL_MASK, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) warp_tot[w] = x;
        __syncthreads();
        if (w == 0) {
            ll t = warp_tot[lane];
            for (int o = 1; o < 32; o <<= 1) {
                const ll y = __shfl_up_sync(FULL_MASK, t, o);
                if (lane >= o) t += y;
            }
            warp_tot[lane] = t;
        }
        __syncthreads();
        if (p <= M) base[p] = carry + x - v + (w > 0 ? warp_tot[w - 1] : 0);
        carry += warp_tot[31];
        __syncthreads();
    }
}

/* each collection's root node: the first node of its run (nodes of an
 * empty collection: the empty range at the next one's root) */
__global__ void __launch_bounds__(1024) k_bh_roots(DevCtl *ctl, SimSegs seg, BhTree t, const ll *base)
{
    if (ctl->error) return;
    for (int s = threadIdx.x; s <= seg.nsims; s += blockDim.x) t.sroot[s] = base[t.stree[s]];
}

/* one thread per sorted position: every node that starts there */
__global__ void __launch_bounds__(BH_BLOCK) k_bh_nodes(DevCtl *ctl, SimSegs seg, const ull *keys, const ll *base,
                                                       BhTree t)
{
    if (ctl->error) return;
    const ll M = ctl->bh_count;
    const ll total = ctl->bh_nodes;
    for (ll p = (ll)blockIdx.x * blockDim.x + threadIdx.x; p < M; p += (ll)gridDim.x * blockDim.x) {
        const int r = bh_run_of(t, seg.nsims, p);
        const ll lo = t.stree[r], hi = t.stree[r + 1];
        int d0, d1;
        node_levels(keys, p, lo, hi, d0, d1);
        if (d1 < d0) continue;
        const ull key = keys[p];
        /* the cube of the level-d0 node: descend d0 levels along the key */
        double cx, cy, cz, half;
        bh_root(t, r, cx, cy, cz, half);
        for (int d = 0; d < d0; d++) {
            const unsigned oct = (unsigned)(key >> (3 * (BH_LEVELS - 1 - d))) & 7u;
            const double q = half / 2;
            cx = (oct & 1u) ? cx + q : cx - q;
            cy = (oct & 2u) ? cy + q : cy - q;
            cz = (oct & 4u) ? cz + q : cz - q;
            half = half / 2;
        }
        for (int d = d0; d <= d1; d++) {
            const ll id = base[p] + (d - d0);
            /* end of the body range: the first key of the run past this
             * node's prefix */
            ll end = hi;
            if (d > 0) {
                const int sh = 3 * (BH_LEVELS - d);
                const ull pre = key >> sh;
                ll a = p + 1, b = hi;
                while (a < b) {
                    const ll mid = (a + b) >> 1;
                    if ((keys[mid] >> sh) <= pre)
                        a = mid + 1;
                    else
                        b = mid;
                }
                end = a;
            }
            t.start[id] = (int)p;
            t.end[id] = (int)end;
            t.skip[id] = (int)(end >= M ? total : base[end]);
            t.flags[id] = (end - p == 1 || d == BH_LEVELS) ? BH_F_LEAF : 0u;
            t.cx[id] = cx;
            t.cy[id] = cy;
            t.cz[id] = cz;
            t.half[id] = half;
            t.fd[id] = make_float4((float)cx, (float)cy, (float)cz, (float)half);
            if (d < d1) {
                const unsigned oct = (unsigned)(key >> (3 * (BH_LEVELS - 1 - d))) & 7u;
                const double q = half / 2;
                cx = (oct & 1u) ? cx + q : cx - q;
                cy = (oct & 2u) ? cy + q : cy - q;
                cz = (oct & 4u) ? cz + q : cz - q;
                half = half / 2;
            }
        }
    }
}

/* ---- 4. masses, from the leaves up ------------------------------------------ */

/* Each node's mass, moments and first body (in array order).  A leaf is one
 * lane's; of a node's children the lane that finishes last (they count
 * themselves in the node's first, which holds no body yet) takes the node, so
 * nothing waits and no sum depends on who is last.  The nodes that a warp has
 * taken are summed eight at a time, a lane for the mass and each moment, over
 * the children in their order: an FP64 add costs the same for one lane as for
 * 32, and one lane a node would spend four times as many.  (The centres of mass
 * are divided out with every lane busy, in the preparation of the walks.)  One
 * launch where each of 22 levels' launches read every node's level: 290 -> 71 us
 * for 131,072 Plummer bodies, 785 -> 313 us for 1,000,003 uniform ones. */
__global__ void __launch_bounds__(BH_BLOCK) k_bh_mass(BodyArrays A, DevCtl *ctl, const unsigned *vals, BhTree t)
{
    if (ctl->error) return;
    const ll total = ctl->bh_nodes;
    const int lane = threadIdx.x & 31, q = lane & 3;
    double *const sum = q == 0 ? t.mass : q == 1 ? t.mx : q == 2 ? t.my : t.mz;
    for (ll base = (ll)blockIdx.x * blockDim.x + (threadIdx.x & ~31u); base < total;
         base += (ll)gridDim.x * blockDim.x) {
        int node = (int)base + lane;
        bool done = base + lane < total && (t.flags[base + lane] & BH_F_LEAF);
        if (done) {
            double M = 0, mx = 0, my = 0, mz = 0;
            int first = 0x7fffffff;
            for (int e = t.start[node]; e < t.end[node]; e++) {
                const unsigned k = vals[e];
                const double m = A.m[k];
                M = M + m;
                mx = mx + A.x[k] * m;
                my = my + A.y[k] * m;
                mz = mz + A.z[k] * m;
                if ((int)k < first) first = (int)k;
            }
            t.mass[node] = M;
            t.mx[node] = mx;
            t.my[node] = my;
            t.mz[node] = mz;
            t.first[node] = first;
        }
        for (;;) {
            __threadfence(); /* this node's sums before its count */
            __syncwarp();
            int p = done ? t.parent[node] : -1;
            if (p >= 0 && atomicAdd(&t.first[p], 1) != (int)t.ccount[p] - 1) p = -1;
            unsigned todo = __ballot_sync(FULL_MASK, p >= 0);
            if (!todo) break;
            __threadfence(); /* every child's sums after the last count */
            __syncwarp();
            while (todo) {
                unsigned m = todo; /* the lane>>2-th of the nodes left */
                for (int g = 0; g < (lane >> 2); g++) m &= m - 1u;
                const int id = __shfl_sync(FULL_MASK, p, m ? __ffs(m) - 1 : 0);
                if (m) {
                    const int stop = t.skip[id];
                    double v = 0;
                    int first = 0x7fffffff;
                    for (int c = id + 1; c < stop; c = t.skip[c]) {
                        v = v + __ldcg(&sum[c]);
                        const int f = __ldcg(&t.first[c]);
                        if (f < first) first = f;
                    }
                    sum[id] = v;
                    if (q == 0) t.first[id] = first;
                }
                for (int g = 0; g < 8; g++) todo &= todo - 1u;
            }
            done = p >= 0;
            node = p;
        }
    }
}

/* The centre of mass of node id, whose mass is M: its moments over its mass,
 * correctly rounded, by integer arithmetic where the operands allow. */
__device__ __forceinline__ void bh_centre(const BhTree &t, ll id, double M, double &cx, double &cy, double &cz)
{
    const double mx = t.mx[id], my = t.my[id], mz = t.mz[id];
    const uint64_t bm = nbx_bits(M), bx = nbx_bits(mx), by = nbx_bits(my), bz = nbx_bits(mz);
    if (nbx_root_ok(bm) && nbx_within(bx, 302) && nbx_within(by, 302) && nbx_within(bz, 302)) {
        const nbx_div d = nbx_operand(nbx_sqrt(bm));
        cx = nbx_double(nbx_pack(nbx_quot(nbx_unpack(bx), d)));
        cy = nbx_double(nbx_pack(nbx_quot(nbx_unpack(by), d)));
        cz = nbx_double(nbx_pack(nbx_quot(nbx_unpack(bz), d)));
    } else {
        cx = mx / M;
        cy = my / M;
        cz = mz / M;
    }
}

/* A node's flags for the walks.  The reference's running centre is 0 / 0 when
 * the node's first body (in array order) is massless, and stays NaN. */
__device__ __forceinline__ unsigned bh_walk_flags(const BodyArrays &A, const BhTree &t, ll id)
{
    return t.flags[id] | (A.m[t.first[id]] == 0 ? BH_F_NAN_CM : 0u);
}

/* ---- 5. forces ------------------------------------------------------------- */

/* accumForce's point-mass term, octree.go:286-292 */
__device__ __forceinline__ void bh_term(double gm_i, double M, double dx, double dy, double dz, double &fx,
                                        double &fy, double &fz)
{
    const double distSq = dx * dx + dy * dy + dz * dz + BH_SOFTENING * BH_SOFTENING;
    const double dist = sqrt(distSq);
    const double force = gm_i * M / distSq;
    fx += force * dx / dist;
    fy += force * dy / dist;
    fz += force * dz / dist;
}

enum { BHW_DROP = 0, BHW_OPEN = 1, BHW_ACCEPT = 2, BHW_MIXED = 3, BHW_BUCKET = 4 };

__device__ __forceinline__ float warp_minf(float v)
{
    for (int o = 16; o > 0; o >>= 1) v = fminf(v, __shfl_xor_sync(FULL_MASK, v, o));
    return v;
}

/* exclusive prefix of v (0..15) over the lanes and the warp's total */
__device__ __forceinline__ int warp_prefix4(int v, unsigned lt, int &total)
{
    int x = 0;
    total = 0;
#pragma unroll
    for (int b = 0; b < 4; b++) {
        const unsigned m = __ballot_sync(FULL_MASK, (v >> b) & 1);
        x += __popc(m & lt) << b;
        total += __popc(m) << b;
    }
    return x;
}

/* Where the walk finds a node: the children of a node take consecutive
 * slots, so a visit that opens it goes on with one address and a count.
 * Slots 0 .. nsims - 1 are the roots'; the others are handed out a warp of
 * nodes at a time (which children lie where does not matter to the sums, only
 * the order among siblings does, and that is theirs). */
__global__ void __launch_bounds__(BH_BLOCK) k_bh_children(DevCtl *ctl, SimSegs seg, BhTree t)
{
    if (ctl->error) return;
    const ll total = ctl->bh_nodes;
    const int lane = threadIdx.x & 31;
    for (ll base = (ll)blockIdx.x * blockDim.x + (threadIdx.x & ~31u); base < total;
         base += (ll)gridDim.x * blockDim.x) {
        const ll id = base + lane;
        int nc = 0, child[8];
        if (id < total && !(t.flags[id] & BH_F_LEAF)) {
            const int stop = t.skip[id];
            int c = (int)id + 1;
#pragma unroll
            for (int q = 0; q < 8; q++) {
                child[q] = c;
                if (c < stop) {
                    nc++;
                    c = t.skip[c];
                }
            }
        }
        int x = nc;
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(FULL_MASK, x, o);
            if (lane >= o) x += y;
        }
        unsigned at = 0;
        if (lane == 31) at = atomicAdd(&ctl->bh_slots, (unsigned)x);
        at = __shfl_sync(FULL_MASK, at, 31);
        if (id < total) {
            const int first = (int)at + seg.nsims + x - nc;
            t.cbase[id] = first;
            t.ccount[id] = (unsigned char)nc;
            t.first[id] = 0; /* k_bh_mass counts the children that are done here */
#pragma unroll
            for (int q = 0; q < 8; q++)
                if (q < nc) {
                    t.slot[child[q]] = first + q;
                    t.parent[child[q]] = (int)id;
                }
        }
    }
    for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < seg.nsims; s += gridDim.x * blockDim.x)
        if (t.sroot[s] < t.sroot[s + 1]) {
            t.slot[t.sroot[s]] = s;
            t.parent[t.sroot[s]] = -1;
        }
}

/* Group g holds sorted positions [p0, p1) of collection s: the groups of a
 * collection start at its first sorted position, 32 bodies each, so a
 * collection's groups are those it would have alone. */
__device__ __forceinline__ void bh_group(const BhTree &t, int nsims, int g, int &s, ll &p0, ll &p1)
{
    s = nbg_sim_of(t.sgrp, nsims, g);
    p0 = t.stree[s] + 32ll * (g - t.sgrp[s]);
    p1 = p0 + 32 < t.stree[s + 1] ? p0 + 32 : t.stree[s + 1];
}

/* every node's records for the FP64 walk, in its slot: centre of mass as hi/lo
 * floats with the squared opening distance (zero when out of FP32's range:
 * then the bodies decide in FP64), and centre, mass and half size as doubles */
#define BH_F_EMPTY 4u /* no mass below */
__global__ void __launch_bounds__(BH_BLOCK) k_bh_prep64(BodyArrays A, DevCtl *ctl, BhTree t)
{
    if (ctl->error) return;
    const ll total = ctl->bh_nodes;
    for (ll id = (ll)blockIdx.x * blockDim.x + threadIdx.x; id < total; id += (ll)gridDim.x * blockDim.x) {
        const int slot = t.slot[id];
        const double M = t.mass[id], half = t.half[id];
        double cx = 0.0, cy = 0.0, cz = 0.0;
        if (M != 0) bh_centre(t, id, M, cx, cy, cz);
        const float hx = (float)cx, hy = (float)cy, hz = (float)cz;
        const double o = 2 * half / BH_THETA, o2 = o * o;
        t.fa[slot] = make_float4(hx, hy, hz, o2 > 1e-30 && o2 < 1e37 ? (float)o2 : 0.f);
        t.fb[slot] = make_float4((float)(cx - (double)hx), (float)(cy - (double)hy), (float)(cz - (double)hz), 0.f);
        t.fc[slot] = make_int4(t.cbase[id],
                               (int)t.ccount[id] | ((int)(bh_walk_flags(A, t, id) | (M == 0 ? BH_F_EMPTY : 0u)) << 8),
                               t.start[id], t.end[id]);
        t.rec[2 * (ll)slot] = make_double2(cx, cy);
        t.rec[2 * (ll)slot + 1] = make_double2(cz, M);
        t.shalf[slot] = half;
    }
}

/* a node of mass M at (dx, dy, dz) from the body, s the softened squared
 * distance: the term with the ordinary operators */
__device__ __noinline__ void bh_term_plain(double gm, double M, double dx, double dy, double dz, double s, double &ex,
                                           double &ey, double &ez)
{
    const double dist = sqrt(s);
    const double force = gm * M / s;
    ex = force * dx / dist;
    ey = force * dy / dist;
    ez = force * dz / dist;
}

/* the bodies of a leaf at the deepest level, each a leaf of its own */
__device__ __noinline__ int bh_bucket64(const BodyArrays &A, const unsigned *vals, int s, int e, unsigned k, double x,
                                        double y, double z, double gm, double &fx, double &fy, double &fz)
{
    int cnt = 0;
    for (int q = s; q < e; q++) {
        const unsigned j = vals[q];
        const double mj = A.m[j];
        if (j == k || mj == 0) continue;
        bh_term(gm, mj, A.x[j] * mj / mj - x, A.y[j] * mj / mj - y, A.z[j] * mj / mj - z, fx, fy, fz);
        cnt++;
    }
    return cnt;
}

#define B64_STACK 256
#define B64_SPARE 32
#define B64_LIST 32
struct alignas(16) Bh64Warp {
    uint2 stack[B64_STACK]; /* runs of siblings: (first slot, the lanes that have not accepted an ancestor) */
    double x[B64_LIST], y[B64_LIST], z[B64_LIST], m[B64_LIST]; /* accepted nodes waiting to be summed */
    unsigned mask[B64_LIST];
    unsigned char run[B64_STACK];
};

/* The reference's opening test of one body and node. */
__device__ __noinline__ bool bh_accepts(double dx, double dy, double dz, double half)
{
    const double dist = sqrt(dx * dx + dy * dy + dz * dz + BH_SOFTENING * BH_SOFTENING);
    return 2 * half / dist < BH_THETA;
}

/* The FP64 walk.  A CTA's four warps take a group of 32 bodies, one body a
 * lane, and walk the tree as the mixed walk does (below): 32 nodes at a time
 * are tested against the group's box in FP32, and nodes the box straddles
 * against each body.  The FP32 tests decide all but the bodies within a part
 * in 2^18 of a node's opening distance, which take the reference's test in
 * FP64.  Every warp makes the whole walk; accepted nodes go to the four in
 * turn, and each adds its own with the reference's expressions, one node at a
 * time, every lane its body: root, quotients and products on the integer
 * pipes, correctly rounded (nbg_exact.h).  A body's terms are those of a walk
 * of its own, summed in the group's order.
 *
 * A thread walking alone spent its time on the FP64 pipe, 85 operations a
 * term with the compiler's root and divisions, and on the walks of its warp's
 * other lanes; now a term takes 12 operations of 19 cycles, with 160 cycles of
 * integer issue beside them.  Tree pass: 2,000 Plummer bodies 8.9 -> 1.24 ms,
 * 30,011 bodies 29.3 -> 7.0 ms, 131,072 bodies 133 -> 28.9 ms.  Dealing runs
 * of nodes to the warps, as the mixed walk does, left one warp most of the
 * near nodes, and so most of the time (19.9 ms at 30,011 bodies); conversions
 * between FP64 and FP32 run on the FP64 pipe too, so the records hold both
 * (13.9 ms when the walk converted them). */
__global__ void __launch_bounds__(BHW_BLOCK, 5) k_bh_force(const __grid_constant__ BodyArrays A, DevCtl *ctl,
                                                           SimSegs seg, const unsigned *vals,
                                                           const __grid_constant__ BhTree t)
{
    __shared__ Bh64Warp ws[BHW_TEAM];
    __shared__ double red[BHW_TEAM - 1][3][32];
    __shared__ int s_grp;
    if (ctl->error) return;
    if (ctl->bh_nodes <= 0) return;
    const int lane = threadIdx.x & 31, wi = threadIdx.x >> 5;
    Bh64Warp &w = ws[wi];
    const unsigned lt = (1u << lane) - 1u;
    const ll groups = t.sgrp[seg.nsims];
    const float soft2 = (float)(BH_SOFTENING * BH_SOFTENING);
    unsigned long long all_terms = 0;
    for (;;) {
        if (threadIdx.x == 0) s_grp = (int)atomicAdd(&ctl->bh_next, 1u);
        __syncthreads();
        const int grp = s_grp;
        __syncthreads();
        if ((ll)grp >= groups) break;
        int r;
        ll p0, p1;
        bh_group(t, seg.nsims, grp, r, p0, p1);
        const ll p = p0 + lane;
        unsigned k = 0;
        bool have = p < p1;
        if (have) {
            k = vals[p];
            have = !(A.flags[k] & NBG_F_IS_SUN); /* k_bh_sun */
        }
        const unsigned every = __ballot_sync(FULL_MASK, have);
        if (!every) continue; /* the same in every warp */
        const double bx = have ? A.x[k] : 0.0, by = have ? A.y[k] : 0.0, bz = have ? A.z[k] : 0.0;
        const double gm = have ? NBG_G * A.m[k] : 0.0;
        const nbx_num gmu = nbx_unpack(nbx_bits(gm));
        const bool gm_ok = nbx_mass_ok(nbx_bits(gm));
        /* the group's box in FP32, widened past every rounding, and the
         * body's position as hi/lo floats for its own tests */
        float gx, gy, gz, ex, ey, ez;
        const float v[3] = {(float)bx, (float)by, (float)bz};
        const float vl[3] = {(float)(bx - (double)v[0]), (float)(by - (double)v[1]), (float)(bz - (double)v[2])};
        {
            float g3[3], e3[3];
#pragma unroll
            for (int c = 0; c < 3; c++) {
                const float lo = warp_minf(have ? v[c] : 3e38f), hi = -warp_minf(have ? -v[c] : 3e38f);
                g3[c] = 0.5f * lo + 0.5f * hi;
                e3[c] = fmaxf(hi - g3[c], g3[c] - lo) + 0x1p-20f * fmaxf(fabsf(lo), fabsf(hi));
            }
            gx = g3[0], gy = g3[1], gz = g3[2];
            ex = e3[0], ey = e3[1], ez = e3[2];
        }
        double fx = 0.0, fy = 0.0, fz = 0.0;
        unsigned terms = 0;
        int cl = 0, top = 1;
        unsigned turn = 0; /* nodes accepted so far; warp wi takes those with turn % BHW_TEAM == wi */
        if (lane == 0) {
            w.stack[0] = make_uint2((unsigned)r, every);
            w.run[0] = 1;
        }
        __syncwarp();
        /* the listed nodes' terms */
        auto flush = [&]() {
#pragma unroll 1
            for (int q = 0; q < cl; q++) {
                const double dx = w.x[q] - bx, dy = w.y[q] - by, dz = w.z[q] - bz;
                const double M = w.m[q];
                const bool mine = (w.mask[q] >> lane) & 1u;
                const uint64_t ux = nbx_bits(dx), uy = nbx_bits(dy), uz = nbx_bits(dz);
                const double s = dx * dx + dy * dy + dz * dz + BH_SOFTENING * BH_SOFTENING;
                const nbx_root root = nbx_sqrt(nbx_bits(s));
                const nbx_num f = nbx_quot(nbx_mul(gmu, nbx_unpack(nbx_bits(M))), nbx_operand(root));
                double tx = nbx_zero(ux) ? 0.0 : nbx_double(nbx_pack(nbx_quot(nbx_mul(f, nbx_unpack(ux)), root.r)));
                double ty = nbx_zero(uy) ? 0.0 : nbx_double(nbx_pack(nbx_quot(nbx_mul(f, nbx_unpack(uy)), root.r)));
                double tz = nbx_zero(uz) ? 0.0 : nbx_double(nbx_pack(nbx_quot(nbx_mul(f, nbx_unpack(uz)), root.r)));
                if (mine) {
                    if (!(nbx_diff_ok(ux) && nbx_diff_ok(uy) && nbx_diff_ok(uz) && gm_ok && nbx_mass_ok(nbx_bits(M))))
                        bh_term_plain(gm, M, dx, dy, dz, s, tx, ty, tz);
                    fx += tx;
                    fy += ty;
                    fz += tz;
                    terms++;
                }
            }
            cl = 0;
            __syncwarp();
        };
        while (top > 0) {
            /* the next 32 nodes, as in the mixed walk */
            int take = B64_STACK - B64_SPARE - top;
            take = take > 32 ? 32 : take < 1 ? 1 : take;
            int cls = BHW_DROP, nc = 0, s = 0, e = 0, cb = 0;
            unsigned mask = 0;
            unsigned slot = 0;
            float4 na = make_float4(0.f, 0.f, 0.f, 0.f), nb = na;
            int4 nd = make_int4(0, 0, 0, 0);
            {
                uint2 en = make_uint2(0u, 0u);
                int rn = 0;
                if (lane < top) {
                    en = w.stack[top - 1 - lane];
                    rn = w.run[top - 1 - lane];
                }
                int tot;
                const int x = warp_prefix4(rn, lt, tot);
                if (take > tot) take = tot;
                const unsigned mark = __reduce_or_sync(FULL_MASK, rn > 0 && x < take ? 1u << x : 0u);
                const unsigned m = mark & (0xffffffffu >> (31 - lane));
                const int from = __popc(m) - 1, off = lane - (31 - __clz(m));
                slot = __shfl_sync(FULL_MASK, en.x, from) + (unsigned)off;
                mask = __shfl_sync(FULL_MASK, en.y, from);
                if (lane < take) {
                    na = t.fa[slot];
                    nb = t.fb[slot];
                    nd = t.fc[slot];
                }
                if (x < take && x + rn > take) {
                    w.stack[top - 1 - lane] = make_uint2(en.x + (unsigned)(take - x), en.y);
                    w.run[top - 1 - lane] = (unsigned char)(x + rn - take);
                }
                top -= __popc(__ballot_sync(FULL_MASK, rn > 0 && x + rn <= take));
            }
            const float o2 = na.w; /* the opening distance squared */
            if (lane < take) {
                cb = nd.x;
                nc = nd.y & 0xff;
                s = nd.z;
                e = nd.w;
                const unsigned fl = (unsigned)nd.y >> 8;
                if (fl & BH_F_EMPTY) {
                    cls = BHW_DROP; /* nothing with mass below: skipped by every body */
                } else if (fl & BH_F_LEAF) {
                    cls = e - s > 1 ? BHW_BUCKET : BHW_ACCEPT;
                    /* a one-body leaf holds sorted position s: not for itself */
                    if (cls == BHW_ACCEPT && s >= p0 && s < p0 + 32) mask &= ~(1u << (int)(s - p0));
                } else if (fl & BH_F_NAN_CM) {
                    cls = BHW_OPEN;
                } else {
                    const float ux = fabsf(na.x - gx), uy = fabsf(na.y - gy), uz = fabsf(na.z - gz);
                    const float mx = ex + 0x1p-20f * fabsf(na.x), my = ey + 0x1p-20f * fabsf(na.y);
                    const float mz = ez + 0x1p-20f * fabsf(na.z);
                    const float nx = fmaxf(ux - mx, 0.f), ny = fmaxf(uy - my, 0.f), nz = fmaxf(uz - mz, 0.f);
                    const float qx = ux + mx, qy = uy + my, qz = uz + mz;
                    const float rn = nx * nx + ny * ny + nz * nz, rf = qx * qx + qy * qy + qz * qz + soft2;
                    cls = o2 == 0.f ? BHW_MIXED
                          : rn * (1.0f - 0x1p-18f) > o2 && rn < 1e37f ? BHW_ACCEPT
                          : rf * (1.0f + 0x1p-18f) < o2 ? BHW_OPEN : BHW_MIXED;
                }
            }
            __syncwarp();
            {
                const unsigned om = __ballot_sync(FULL_MASK, cls == BHW_OPEN);
                if (cls == BHW_OPEN) {
                    const int at = top + __popc(om & lt);
                    w.stack[at] = make_uint2((unsigned)cb, mask);
                    w.run[at] = (unsigned char)nc;
                }
                top += __popc(om);
            }
            /* the nodes the box straddles: each body's own test */
            const unsigned mm = __ballot_sync(FULL_MASK, cls == BHW_MIXED);
            {
                for (unsigned mq = mm; mq; mq &= mq - 1u) {
                    const int src = __ffs(mq) - 1;
                    const float dx = (__shfl_sync(FULL_MASK, na.x, src) - v[0]) + (__shfl_sync(FULL_MASK, nb.x, src) - vl[0]);
                    const float dy = (__shfl_sync(FULL_MASK, na.y, src) - v[1]) + (__shfl_sync(FULL_MASK, nb.y, src) - vl[1]);
                    const float dz = (__shfl_sync(FULL_MASK, na.z, src) - v[2]) + (__shfl_sync(FULL_MASK, nb.z, src) - vl[2]);
                    const float q2 = __shfl_sync(FULL_MASK, o2, src);
                    const unsigned mk = __shfl_sync(FULL_MASK, mask, src);
                    const float r2 = dx * dx + dy * dy + dz * dz + soft2;
                    const bool mine = (mk >> lane) & 1u;
                    const bool in = q2 != 0.f && r2 < 1e37f;
                    bool accept = in && r2 * (1.0f - 0x1p-18f) > q2;
                    const bool sure = accept || (in && r2 * (1.0f + 0x1p-18f) < q2);
                    if (__any_sync(FULL_MASK, mine && !sure)) {
                        const ll sl = (ll)__shfl_sync(FULL_MASK, slot, src);
                        if (!sure) {
                            const double2 ra = t.rec[2 * sl], rb = t.rec[2 * sl + 1];
                            accept = bh_accepts(ra.x - bx, ra.y - by, rb.x - bz, t.shalf[sl]);
                        }
                    }
                    const unsigned am = __ballot_sync(FULL_MASK, mine && accept);
                    const unsigned om = mk & ~am;
                    if (lane == src) {
                        if (om) {
                            w.stack[top] = make_uint2((unsigned)cb, om);
                            w.run[top] = (unsigned char)nc;
                        }
                        mask = am;
                        cls = am ? BHW_ACCEPT : BHW_DROP;
                    }
                    top += om ? 1 : 0;
                }
            }
            /* accepted nodes, in turn to the team's warps */
            {
                const unsigned am = __ballot_sync(FULL_MASK, cls == BHW_ACCEPT);
                const bool put = cls == BHW_ACCEPT && ((turn + __popc(am & lt)) % BHW_TEAM) == (unsigned)wi;
                turn += __popc(am);
                const unsigned pm = __ballot_sync(FULL_MASK, put);
                if (cl + __popc(pm) > B64_LIST) flush();
                if (put) {
                    const int at = cl + __popc(pm & lt);
                    const double2 ra = t.rec[2 * (ll)slot], rb = t.rec[2 * (ll)slot + 1];
                    w.x[at] = ra.x;
                    w.y[at] = ra.y;
                    w.z[at] = rb.x;
                    w.m[at] = rb.y;
                    w.mask[at] = mask;
                }
                cl += __popc(pm);
            }
            for (unsigned bm = __ballot_sync(FULL_MASK, cls == BHW_BUCKET && wi == 0); bm; bm &= bm - 1u) {
                const int src = __ffs(bm) - 1;
                const unsigned mk = __shfl_sync(FULL_MASK, mask, src);
                const int bs = __shfl_sync(FULL_MASK, s, src), be = __shfl_sync(FULL_MASK, e, src);
                if ((mk >> lane) & 1u) {
                    double tx = 0.0, ty = 0.0, tz = 0.0;
                    terms += bh_bucket64(A, vals, bs, be, k, bx, by, bz, gm, tx, ty, tz);
                    fx += tx;
                    fy += ty;
                    fz += tz;
                }
                __syncwarp();
            }
            __syncwarp();
        }
        flush();
        /* the team's sums, in warp order */
        if (wi > 0) {
            red[wi - 1][0][lane] = fx;
            red[wi - 1][1][lane] = fy;
            red[wi - 1][2][lane] = fz;
        }
        __syncthreads();
        if (wi == 0 && have) {
            for (int q = 0; q < BHW_TEAM - 1; q++) {
                fx += red[q][0][lane];
                fy += red[q][1][lane];
                fz += red[q][2][lane];
            }
            A.fx[k] = fx;
            A.fy[k] = fy;
            A.fz[k] = fz;
        }
        all_terms += terms;
    }
    /* point-mass terms summed, for the measured work */
    for (int o = 16; o > 0; o >>= 1) all_terms += __shfl_xor_sync(FULL_MASK, all_terms, o);
    if (lane == 0 && all_terms) atomicAdd((unsigned long long *)&ctl->acc_bh_terms, all_terms);
}

/* ---- 5b. the mixed-precision walk --------------------------------------------
 * The same tree and the same acceptance rule in FP32: centres of mass as
 * hi/lo float pairs (so dx = (cm_hi - x_hi) + (cm_lo - x_lo) keeps ~2^-24 of
 * |dx|), masses relative to the root's, the opening test as
 * r^2 > (2 half / theta)^2 on the softened r^2, and the reciprocal square
 * root of the SFU.
 *
 * A group of 32 bodies (neighbours in key order, one per lane) walks the tree
 * together.  The warp keeps a stack of nodes, each with the lanes that have
 * not accepted an ancestor of it, and visits 32 of them at once, one per
 * lane: most nodes lie so far from the group's box (or so close) that all
 * its bodies accept (or open) them, which one bound decides; accepted nodes
 * are listed in shared memory and summed 32 or more at a time, every lane
 * its own body, two nodes per packed instruction.  Only the nodes in between
 * (1,100 of the 7,900 that a group of a 131,072-body Plummer sphere accepts)
 * take each body's own test, with the same expression and rounding as a walk
 * of that body alone, so every body sums the terms it would alone.  Sums are
 * FP32, folded into (hi, lo) pairs after every list: the GB300 FP64 pipe is
 * 1/64 of the FP32 rate.
 *
 * A walk that took one node at a time for the whole warp was bound by the
 * latency of its node loads (issue slots 25 % busy).  The walk of a 131,072-
 * body Plummer sphere went from 5.0 to 1.54 ms, of 10^6 uniform bodies from
 * 20.3 to 7.2 ms.  What bounds it now is issue and, with a group to a warp,
 * groups of uneven cost: 263,000 instructions a group before the lists were
 * split into far and near ones, 60 % of them in the sums. */
/* every node's record for the walk, in its slot */
__global__ void __launch_bounds__(BH_BLOCK) k_bh_prep_mixed(BodyArrays A, DevCtl *ctl, SimSegs seg, BhTree t)
{
    if (ctl->error) return;
    const ll total = ctl->bh_nodes;
    if (total <= 0) return;
    ll root = -1;
    double inv_root = 0.0;
    for (ll id = (ll)blockIdx.x * blockDim.x + threadIdx.x; id < total; id += (ll)gridDim.x * blockDim.x) {
        /* masses relative to the root of the node's own tree */
        const ll r = t.sroot[nbg_sim_of(t.sroot, seg.nsims, id)];
        if (r != root) {
            const double mroot = t.mass[r];
            inv_root = mroot != 0 ? 1.0 / mroot : 0.0;
            root = r;
        }
        const double M = t.mass[id];
        float4 a = make_float4(0.f, 0.f, 0.f, 0.f), b = make_float4(0.f, 0.f, 0.f, 0.f);
        if (M != 0) {
            double cx, cy, cz;
            bh_centre(t, id, M, cx, cy, cz);
            a.x = (float)cx;
            a.y = (float)cy;
            a.z = (float)cz;
            b.x = (float)(cx - (double)a.x);
            b.y = (float)(cy - (double)a.y);
            b.z = (float)(cz - (double)a.z);
            a.w = (float)(M * inv_root);
            const double o = 2 * t.half[id] / BH_THETA;
            b.w = (float)(o * o);
        }
        /* A centre of mass past FP32's range (or with an infinite moment or
         * mass) is at no distance from any body: the acceptance test opens the
         * node for every one, and a leaf's term is NaN.  Flagged here, so that
         * the walk neither bounds the distance nor adds the term for bodies
         * that accepted an ancestor. */
        unsigned fl = bh_walk_flags(A, t, id);
        if (!(fabsf(a.x) <= BH_FLT_MAX && fabsf(a.y) <= BH_FLT_MAX && fabsf(a.z) <= BH_FLT_MAX))
            fl |= (fl & BH_F_LEAF) ? BH_F_FAR_OUT : BH_F_NAN_CM;
        const int slot = t.slot[id];
        t.fa[slot] = a;
        t.fb[slot] = b;
        t.fc[slot] = make_int4(t.cbase[id], (int)t.ccount[id] | ((int)fl << 8), t.start[id], t.end[id]);
    }
}

/* (hi, lo) += v with the rounding error of hi + v kept in lo (TwoSum) */
__device__ __forceinline__ void fold2(float &hi, float &lo, float v)
{
    const float s = hi + v;
    const float bb = s - hi;
    const float e = (hi - (s - bb)) + (v - bb);
    hi = s;
    lo += e;
}

__device__ __forceinline__ float bh_rsqrt(float x)
{
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

/* the terms of a leaf at the deepest level holding bodies [s, e), or of one
 * body past FP32's range (rare; kept out of the walk's registers) */
__device__ __noinline__ int bucket_terms(const BodyArrays &A, const unsigned *vals, int s, int e, unsigned k, float xh,
                                         float yh, float zh, float xl, float yl, float zl, float soft2, double mroot,
                                         float &ax, float &ay, float &az)
{
    int cnt = 0;
    for (int q = s; q < e; q++) {
        const unsigned j = vals[q];
        const double mj = A.m[j];
        if (j == k || mj == 0) continue;
        if (e - s == 1) {
            ax = ay = az = __int_as_float(0x7fc00000);
            return 1;
        }
        const float ex = (float)(A.x[j] - (double)xh - (double)xl);
        const float ey = (float)(A.y[j] - (double)yh - (double)yl);
        const float ez = (float)(A.z[j] - (double)zh - (double)zl);
        const float q2 = ex * ex + ey * ey + ez * ez + soft2;
        const float inv = bh_rsqrt(q2);
        const float w = (float)(mj / mroot) * inv * inv * inv;
        ax += w * ex;
        ay += w * ey;
        az += w * ez;
        cnt++;
    }
    return cnt;
}

/* one warp's working set in shared memory */
/* runs of sibling nodes still to visit.  Full stacks take nodes one by one:
 * 384 single nodes in place of runs of up to eight made the walk twice as
 * long, 1,024 still 10 % longer than 2,048. */
#ifndef BHW_STACK
#define BHW_STACK 256
#endif
#define BHW_SPARE 32 /* of them kept for taking one node at a time: one a level, 21 levels */
#define BHW_FAR 64    /* far nodes waiting to be summed */
#define BHW_MIX 32    /* nodes that need each body's own test, waiting */
/* a node counts as far when its centre of mass is this many half extents of
 * the group's box away: re-centred on the box, its coordinates then carry no
 * more than 1.5 times the rounding of the bodies' distances to it */
#ifndef BHW_FAR_RATIO
#define BHW_FAR_RATIO 3.0f
#endif
struct alignas(16) BhWarp {
    uint2 stack[BHW_STACK]; /* (first slot, the lanes that have not accepted an ancestor) */
    /* far nodes, relative to the box */
    float fx[BHW_FAR + 4], fy[BHW_FAR + 4], fz[BHW_FAR + 4], fm[BHW_FAR + 4];
    unsigned fmask[BHW_FAR + 4];
    /* nodes the bodies may disagree on, and accepted ones close by */
    float hx[BHW_MIX + 4], hy[BHW_MIX + 4], hz[BHW_MIX + 4], m[BHW_MIX + 4];
    float lx[BHW_MIX + 4], ly[BHW_MIX + 4], lz[BHW_MIX + 4], open2[BHW_MIX + 4];
    unsigned mask[BHW_MIX + 4];
    int cb[BHW_MIX], nc[BHW_MIX];
    unsigned char run[BHW_STACK]; /* nodes of each run */
};
/* FP32 partial sums and the (hi, lo) pairs they are folded into */
struct BhSum {
    float2 ax, ay, az;
    float hx, lx, hy, ly, hz, lz;
    __device__ __forceinline__ void term(const float2 &m, const float2 &r2, const float2 &dx, const float2 &dy,
                                         const float2 &dz)
    {
        const float2 inv = make_float2(bh_rsqrt(r2.x), bh_rsqrt(r2.y));
        const float2 wt = __fmul2_rn(__fmul2_rn(m, inv), __fmul2_rn(inv, inv));
        ax = __ffma2_rn(wt, dx, ax);
        ay = __ffma2_rn(wt, dy, ay);
        az = __ffma2_rn(wt, dz, az);
    }
    __device__ __forceinline__ void fold()
    {
        fold2(hx, lx, ax.x + ax.y);
        fold2(hy, ly, ay.x + ay.y);
        fold2(hz, lz, az.x + az.y);
        ax = ay = az = make_float2(0.f, 0.f);
    }
};

template <int MINB>
__global__ void __launch_bounds__(BHW_BLOCK, MINB) k_bh_force_mixed(const __grid_constant__ BodyArrays A, DevCtl *ctl,
                                                                 SimSegs seg, const unsigned *vals,
                                                                 const __grid_constant__ BhTree t)
{
    __shared__ BhWarp ws[BHW_TEAM];
    __shared__ float red[BHW_TEAM - 1][6][32];
    __shared__ int s_unit;
    if (ctl->error) return;
    if (ctl->bh_nodes <= 0) return;
    const int lane = threadIdx.x & 31, wi = threadIdx.x >> 5;
    BhWarp &w = ws[wi];
    const unsigned lt = (1u << lane) - 1u;
    const ll units = t.sunit[seg.nsims];
    const float soft2 = (float)(BH_SOFTENING * BH_SOFTENING);
    const float2 s2 = make_float2(soft2, soft2);
    const float4 zero4 = make_float4(0.f, 0.f, 0.f, 0.f);
    unsigned long long all_terms = 0;
    for (;;) {
        if (threadIdx.x == 0) s_unit = (int)atomicAdd(&ctl->bh_next, 1u);
        __syncthreads();
        const int unit = s_unit;
        __syncthreads();
        if ((ll)unit >= units) break;
        const int r = nbg_sim_of(t.sunit, seg.nsims, unit);
        const ll n_r = t.scount[r];
        const bool solo = n_r >= BHW_SOLO_MIN;
        const ll g = solo ? BHW_TEAM * (unit - t.sunit[r]) + wi : unit - t.sunit[r];
        const ll p0 = t.stree[r] + 32 * g, p1 = p0 + 32 < t.stree[r + 1] ? p0 + 32 : t.stree[r + 1];
        const ll p = p0 + lane;
        unsigned k = 0;
        bool have = p < p1;
        if (have) {
            k = vals[p];
            have = !(A.flags[k] & NBG_F_IS_SUN); /* k_bh_sun */
        }
        const unsigned every = __ballot_sync(FULL_MASK, have);
        if (!every) continue; /* solo warps meet at the next unit; a team's agree */
        float2 xh, yh, zh, xl, yl, zl; /* (-hi, -hi) and (-lo, -lo) of the lane's body */
        float2 xr, yr, zr;             /* minus its offset from the box's centre */
        float gx, gy, gz, ex, ey, ez, far2;
        {
            float vh[3] = {0.f, 0.f, 0.f}, vl[3] = {0.f, 0.f, 0.f};
            if (have) {
                const double x = A.x[k], y = A.y[k], z = A.z[k];
                vh[0] = (float)x;
                vh[1] = (float)y;
                vh[2] = (float)z;
                vl[0] = (float)(x - (double)vh[0]);
                vl[1] = (float)(y - (double)vh[1]);
                vl[2] = (float)(z - (double)vh[2]);
            }
            /* the group's box: centre g, half extents e, widened past the
             * rounding of the positions and of the distances to it */
            float g3[3], e3[3], o3[3];
#pragma unroll
            for (int c = 0; c < 3; c++) {
                const float lo = warp_minf(have ? vh[c] : 3e38f), hi = -warp_minf(have ? -vh[c] : 3e38f);
                g3[c] = 0.5f * lo + 0.5f * hi;
                e3[c] = fmaxf(hi - g3[c], g3[c] - lo) + 0x1p-20f * fmaxf(fabsf(lo), fabsf(hi));
                o3[c] = (vh[c] - g3[c]) + vl[c];
            }
            gx = g3[0], gy = g3[1], gz = g3[2];
            ex = e3[0], ey = e3[1], ez = e3[2];
            far2 = (BHW_FAR_RATIO * BHW_FAR_RATIO) * (ex * ex + ey * ey + ez * ez);
            xh = make_float2(-vh[0], -vh[0]);
            yh = make_float2(-vh[1], -vh[1]);
            zh = make_float2(-vh[2], -vh[2]);
            xl = make_float2(-vl[0], -vl[0]);
            yl = make_float2(-vl[1], -vl[1]);
            zl = make_float2(-vl[2], -vl[2]);
            xr = make_float2(-o3[0], -o3[0]);
            yr = make_float2(-o3[1], -o3[1]);
            zr = make_float2(-o3[2], -o3[2]);
        }
        BhSum b;
        b.ax = b.ay = b.az = make_float2(0.f, 0.f);
        b.hx = b.lx = b.hy = b.ly = b.hz = b.lz = 0.f;
        unsigned terms = 0;
        int cf = 0, cm = 0; /* nodes in the two lists */
        int top = 1;
        /* until the walk is dealt out, every warp of a team walks the same
         * top of the tree, and only the first keeps its terms */
        bool dealt = solo;
        if (lane == 0) {
            w.stack[0] = make_uint2((unsigned)r, every);
            w.run[0] = 1;
        }
        __syncwarp();
        /* the far list's terms, two per packed instruction */
        auto flush = [&]() {
            if (lane < 3) {
                const int at = cf + lane; /* up to a multiple of four with nothing */
                w.fx[at] = w.fy[at] = w.fz[at] = w.fm[at] = 0.f;
                w.fmask[at] = every;
            }
            __syncwarp();
#pragma unroll 1
            for (int q = 0; q < cf; q += 4) {
                const float4 X = *(const float4 *)&w.fx[q], Y = *(const float4 *)&w.fy[q];
                const float4 Z = *(const float4 *)&w.fz[q];
                float4 M = *(const float4 *)&w.fm[q];
                const uint4 K = *(const uint4 *)&w.fmask[q];
                if ((K.x & K.y & K.z & K.w) != every) {
                    M.x = (K.x >> lane) & 1u ? M.x : 0.f;
                    M.y = (K.y >> lane) & 1u ? M.y : 0.f;
                    M.z = (K.z >> lane) & 1u ? M.z : 0.f;
                    M.w = (K.w >> lane) & 1u ? M.w : 0.f;
                }
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    const float2 dx = __fadd2_rn(h ? make_float2(X.z, X.w) : make_float2(X.x, X.y), xr);
                    const float2 dy = __fadd2_rn(h ? make_float2(Y.z, Y.w) : make_float2(Y.x, Y.y), yr);
                    const float2 dz = __fadd2_rn(h ? make_float2(Z.z, Z.w) : make_float2(Z.x, Z.y), zr);
                    const float2 r2 = __ffma2_rn(dz, dz, __ffma2_rn(dy, dy, __ffma2_rn(dx, dx, s2)));
                    b.term(h ? make_float2(M.z, M.w) : make_float2(M.x, M.y), r2, dx, dy, dz);
                }
            }
            b.fold();
            cf = 0;
            __syncwarp();
        };
        /* the second list: each body's own test, with the precise distance;
         * the children of the nodes that some body opens go on the stack */
        auto settle = [&]() {
            if (lane < 3) {
                const int at = cm + lane;
                w.hx[at] = w.hy[at] = w.hz[at] = w.m[at] = w.lx[at] = w.ly[at] = w.lz[at] = w.open2[at] = 0.f;
                w.mask[at] = 0u;
            }
            __syncwarp();
            unsigned open = 0, tm = 0;
#pragma unroll 1
            for (int q = 0; q < cm; q += 2) {
                const float2 X = *(const float2 *)&w.hx[q], Y = *(const float2 *)&w.hy[q], Z = *(const float2 *)&w.hz[q];
                const float2 U = *(const float2 *)&w.lx[q], V = *(const float2 *)&w.ly[q], W = *(const float2 *)&w.lz[q];
                const float2 M = *(const float2 *)&w.m[q], O = *(const float2 *)&w.open2[q];
                const uint2 K = *(const uint2 *)&w.mask[q];
                const float2 dx = __fadd2_rn(__fadd2_rn(X, xh), __fadd2_rn(U, xl));
                const float2 dy = __fadd2_rn(__fadd2_rn(Y, yh), __fadd2_rn(V, yl));
                const float2 dz = __fadd2_rn(__fadd2_rn(Z, zh), __fadd2_rn(W, zl));
                /* rounded as the acceptance rule states it: each square, the
                 * sums left to right, the softening last */
                const float2 r2 = __fadd2_rn(
                    __fadd2_rn(__fadd2_rn(__fmul2_rn(dx, dx), __fmul2_rn(dy, dy)), __fmul2_rn(dz, dz)), s2);
                const bool k0 = (K.x >> lane) & 1u, k1 = (K.y >> lane) & 1u;
                const bool a0 = k0 && r2.x > O.x, a1 = k1 && r2.y > O.y;
                const unsigned o0 = __ballot_sync(FULL_MASK, k0 && !a0), o1 = __ballot_sync(FULL_MASK, k1 && !a1);
                if (lane == q) open = o0;
                if (lane == q + 1) open = o1;
                tm += (unsigned)a0 + (unsigned)a1;
                b.term(make_float2(a0 ? M.x : 0.f, a1 ? M.y : 0.f), r2, dx, dy, dz);
            }
            b.fold();
            if (dealt || wi == 0) terms += tm;
            const unsigned om = __ballot_sync(FULL_MASK, open != 0u); /* lanes below cm only */
            if (open) {
                const int at = top + __popc(om & lt);
                w.stack[at] = make_uint2((unsigned)w.cb[lane], open);
                w.run[at] = (unsigned char)w.nc[lane];
            }
            top += __popc(om);
            cm = 0;
            __syncwarp();
        };
        for (;;) {
            if (cm > 0 && (top == 0 || !dealt || top + cm + 32 > BHW_STACK - BHW_SPARE)) settle();
            if (!dealt && (top == 0 || top >= 32)) {
                /* the team's warps take every BHW_TEAM-th run */
                int n = 0;
                for (int s0 = 0; s0 < top; s0 += 32 * BHW_TEAM) {
                    const int i = s0 + lane * BHW_TEAM + wi;
                    const uint2 en = i < top ? w.stack[i] : make_uint2(0u, 0u);
                    const unsigned char rn = i < top ? w.run[i] : 0;
                    __syncwarp();
                    if (i < top) {
                        w.stack[n + lane] = en;
                        w.run[n + lane] = rn;
                    }
                    n += __popc(__ballot_sync(FULL_MASK, i < top));
                    __syncwarp();
                }
                top = n;
                dealt = true;
            }
            if (top == 0) break; /* the second list is empty here too */
            /* The next 32 nodes at once, of the topmost runs: lane i reads run
             * i from the top; `mark` has a bit at each run's first node.  Each
             * node leaves at most one run, so a nearly full stack takes fewer,
             * down to one at a time: a descent that adds a run a level. */
            int take = BHW_STACK - BHW_SPARE - top - cm;
            take = take > 32 ? 32 : take < 1 ? 1 : take;
            int cls = BHW_DROP, nc = 0, s = 0, e = 0, cb = 0;
            unsigned mask = 0;
            float4 na = zero4, nb = zero4;
            int4 nd = make_int4(0, 0, 0, 0);
            {
                uint2 en = make_uint2(0u, 0u);
                int rn = 0;
                if (lane < top) {
                    en = w.stack[top - 1 - lane];
                    rn = w.run[top - 1 - lane];
                }
                int tot;
                const int x = warp_prefix4(rn, lt, tot);
                if (take > tot) take = tot;
                const unsigned mark = __reduce_or_sync(FULL_MASK, rn > 0 && x < take ? 1u << x : 0u);
                const unsigned m = mark & (0xffffffffu >> (31 - lane));
                const int from = __popc(m) - 1, off = lane - (31 - __clz(m));
                const unsigned slot = __shfl_sync(FULL_MASK, en.x, from) + (unsigned)off;
                mask = __shfl_sync(FULL_MASK, en.y, from);
                if (lane < take) {
                    na = t.fa[slot];
                    nb = t.fb[slot];
                    nd = t.fc[slot];
                }
                /* the one run taken in part keeps the rest */
                if (x < take && x + rn > take) {
                    w.stack[top - 1 - lane] = make_uint2(en.x + (unsigned)(take - x), en.y);
                    w.run[top - 1 - lane] = (unsigned char)(x + rn - take);
                }
                /* runs of no nodes go too: a body past FP32's range, whose
                 * distances are NaN, opens accepted nodes, which have no
                 * children here */
                top -= __popc(__ballot_sync(FULL_MASK, lane < top && x + rn <= take));
            }
            if (cf >= 32) flush(); /* while those loads are in flight */
            bool isfar = false;
            if (lane < take) {
                cb = nd.x;
                nc = nd.y & 0xff;
                s = nd.z;
                e = nd.w;
                const unsigned fl = (unsigned)nd.y >> 8;
                const float ux = na.x - gx, uy = na.y - gy, uz = na.z - gz;
                isfar = ux * ux + uy * uy + uz * uz > far2;
                if (na.w == 0.f) {
                    cls = BHW_DROP; /* nothing with mass below: skipped by every body */
                } else if (fl & BH_F_LEAF) {
                    cls = e - s > 1 || (fl & BH_F_FAR_OUT) ? BHW_BUCKET : BHW_ACCEPT;
                    /* a one-body leaf holds sorted position s: not for itself */
                    if (cls == BHW_ACCEPT && s >= p0 && s < p0 + 32) mask &= ~(1u << (int)(s - p0));
                } else if (fl & BH_F_NAN_CM) {
                    cls = BHW_OPEN;
                } else {
                    /* nearest and farthest the box can be from the centre of
                     * mass, with room for every rounding of the bodies' own
                     * tests: outside both bounds the bodies agree */
                    const float mx = ex + 0x1p-20f * fabsf(na.x), my = ey + 0x1p-20f * fabsf(na.y);
                    const float mz = ez + 0x1p-20f * fabsf(na.z);
                    const float nx = fmaxf(fabsf(ux) - mx, 0.f), ny = fmaxf(fabsf(uy) - my, 0.f);
                    const float nz = fmaxf(fabsf(uz) - mz, 0.f);
                    const float fx = fabsf(ux) + mx, fy = fabsf(uy) + my, fz = fabsf(uz) + mz;
                    const float rn = nx * nx + ny * ny + nz * nz, rf = fx * fx + fy * fy + fz * fz + soft2;
                    cls = rn * (1.0f - 0x1p-18f) > nb.w ? BHW_ACCEPT
                          : rf * (1.0f + 0x1p-18f) < nb.w ? BHW_OPEN : BHW_MIXED;
                }
                if (cls == BHW_ACCEPT && !isfar) { /* precise distances, no test, no children */
                    cls = BHW_MIXED;
                    nb.w = -1.f;
                    nc = 0;
                }
            }
            __syncwarp();
            /* opened by every body: its children, for the same bodies */
            {
                const unsigned om = __ballot_sync(FULL_MASK, cls == BHW_OPEN);
                if (cls == BHW_OPEN) {
                    const int at = top + __popc(om & lt);
                    w.stack[at] = make_uint2((unsigned)cb, mask);
                    w.run[at] = (unsigned char)nc;
                }
                top += __popc(om);
            }
            /* accepted by every body, far away: listed */
            const unsigned am = __ballot_sync(FULL_MASK, cls == BHW_ACCEPT && (dealt || wi == 0));
            if ((am >> lane) & 1u) {
                const int at = cf + __popc(am & lt);
                w.fx[at] = (na.x - gx) + nb.x;
                w.fy[at] = (na.y - gy) + nb.y;
                w.fz[at] = (na.z - gz) + nb.z;
                w.fm[at] = na.w;
                w.fmask[at] = mask;
                terms += __popc(mask);
            }
            cf += __popc(am);
            /* each body decides for itself, later */
            const unsigned mm = __ballot_sync(FULL_MASK, cls == BHW_MIXED);
            if (mm) {
                if (cm + __popc(mm) > BHW_MIX) settle();
                if (cls == BHW_MIXED) {
                    const int at = cm + __popc(mm & lt);
                    w.hx[at] = na.x;
                    w.hy[at] = na.y;
                    w.hz[at] = na.z;
                    w.m[at] = dealt || wi == 0 ? na.w : 0.f;
                    w.lx[at] = nb.x;
                    w.ly[at] = nb.y;
                    w.lz[at] = nb.z;
                    w.open2[at] = nb.w;
                    w.mask[at] = mask;
                    w.cb[at] = cb;
                    w.nc[at] = nc;
                }
                cm += __popc(mm);
            }
            /* a leaf at the deepest level holding several bodies, or one past
             * FP32's range */
            for (unsigned bm = __ballot_sync(FULL_MASK, cls == BHW_BUCKET && (dealt || wi == 0)); bm; bm &= bm - 1u) {
                const int src = __ffs(bm) - 1;
                const unsigned mk = __shfl_sync(FULL_MASK, mask, src);
                const int bs = __shfl_sync(FULL_MASK, s, src), be = __shfl_sync(FULL_MASK, e, src);
                if ((mk >> lane) & 1u) {
                    float tx = 0.f, ty = 0.f, tz = 0.f;
                    terms += bucket_terms(A, vals, bs, be, k, -xh.x, -yh.x, -zh.x, -xl.x, -yl.x, -zl.x, soft2,
                                          t.mass[t.sroot[r]], tx, ty, tz);
                    b.ax.x += tx;
                    b.ay.x += ty;
                    b.az.x += tz;
                }
                __syncwarp();
            }
            __syncwarp();
        }
        flush();
        if (!solo) {
            /* the team's sums, in warp order */
            if (wi > 0) {
                red[wi - 1][0][lane] = b.hx;
                red[wi - 1][1][lane] = b.lx;
                red[wi - 1][2][lane] = b.hy;
                red[wi - 1][3][lane] = b.ly;
                red[wi - 1][4][lane] = b.hz;
                red[wi - 1][5][lane] = b.lz;
            }
            __syncthreads();
            if (wi == 0)
                for (int q = 0; q < BHW_TEAM - 1; q++) {
                    fold2(b.hx, b.lx, red[q][0][lane]);
                    fold2(b.hy, b.ly, red[q][2][lane]);
                    fold2(b.hz, b.lz, red[q][4][lane]);
                    b.lx += red[q][1][lane];
                    b.ly += red[q][3][lane];
                    b.lz += red[q][5][lane];
                }
        }
        if (have && (solo || wi == 0)) {
            const double gm = NBG_G * A.m[k] * t.mass[t.sroot[r]];
            A.fx[k] = gm * ((double)b.hx + (double)b.lx);
            A.fy[k] = gm * ((double)b.hy + (double)b.ly);
            A.fz[k] = gm * ((double)b.hz + (double)b.lz);
        }
        all_terms += terms;
    }
    for (int o = 16; o > 0; o >>= 1) all_terms += __shfl_xor_sync(FULL_MASK, all_terms, o);
    if (lane == 0 && all_terms) atomicAdd((unsigned long long *)&ctl->acc_bh_terms, all_terms);
}

/* a sun sums every tree body directly (directForce, octree.go:310-325): each
 * CTA scans a run of bodies for suns, and sums every sun it finds with all
 * its threads, in a fixed-order block reduction */
__global__ void __launch_bounds__(BH_BLOCK) k_bh_sun(BodyArrays A, DevCtl *ctl, SimSegs seg)
{
    __shared__ double red[3][BH_BLOCK];
    __shared__ unsigned s_mask[BH_BLOCK / 32];
    if (ctl->error) return;
    const ll n = ctl->n;
    for (ll base = (ll)blockIdx.x * BH_BLOCK; base < n; base += (ll)gridDim.x * BH_BLOCK) {
        const ll mine = base + threadIdx.x;
        const bool sun = mine < n &&
                         (A.flags[mine] & (NBG_LIVE_MASK | NBG_F_IS_SUN)) == (NBG_F_EXISTS | NBG_F_IS_SUN) &&
                         tree_body(A, mine);
        const unsigned m = __ballot_sync(FULL_MASK, sun);
        if ((threadIdx.x & 31) == 0) s_mask[threadIdx.x >> 5] = m;
        __syncthreads();
        for (int w = 0; w < BH_BLOCK / 32; w++) {
            unsigned bits = s_mask[w];
            while (bits) {
                const int lane = __ffs(bits) - 1;
                bits &= bits - 1;
                const ll k = base + w * 32 + lane;
                const double x = A.x[k], y = A.y[k], z = A.z[k];
                const double gm = NBG_G * A.m[k];
                double fx = 0, fy = 0, fz = 0;
                /* the bodies of the sun's own collection, each thread the
                 * same share of them as if the collection were alone */
                const int sim = nbg_sim_of(seg.off, seg.nsims, k);
                const ll j0 = seg.off[sim], j1 = seg.off[sim + 1];
                for (ll j = j0 + threadIdx.x; j < j1; j += blockDim.x) {
                    if (j == k || (A.flags[j] & NBG_LIVE_MASK) != NBG_F_EXISTS) continue;
                    bh_term(gm, A.m[j], A.x[j] - x, A.y[j] - y, A.z[j] - z, fx, fy, fz);
                }
                red[0][threadIdx.x] = fx;
                red[1][threadIdx.x] = fy;
                red[2][threadIdx.x] = fz;
                __syncthreads();
                for (int st = BH_BLOCK / 2; st > 0; st >>= 1) {
                    if (threadIdx.x < st)
                        for (int q = 0; q < 3; q++) red[q][threadIdx.x] += red[q][threadIdx.x + st];
                    __syncthreads();
                }
                if (threadIdx.x == 0) {
                    A.fx[k] = red[0][0];
                    A.fy[k] = red[1][0];
                    A.fz[k] = red[2][0];
                }
                __syncthreads();
            }
        }
        __syncthreads(); /* s_mask is rewritten for the next run */
    }
}

/* ---- 6. collisions: Compute's second pass as a range query ----------------- */

/* Collided + the event rules for tree body i against body j (j != i) */
__device__ __forceinline__ void bh_test_pair(const BodyArrays &A, DevCtl *ctl, ull *ev_keys, ll ev_cap, ll i,
                                             double xi, double yi, double zi, double ri, unsigned bi, ll j)
{
    const double dx = A.x[j] - xi;
    const double dy = A.y[j] - yi;
    const double dz = A.z[j] - zi;
    const double dist = sqrt(dx * dx + dy * dy + dz * dz);
    const double rj = A.rad[j];
    if (dist <= ri + rj) {
        const int type = nbg_detect_event(bi, NBG_BEHAVIOR(A.flags[j]), ri, rj, dist);
        if (type >= 0) nbg_emit_event(ctl, ev_keys, ev_cap, i, j, type);
    }
}

__global__ void __launch_bounds__(BH_BLOCK) k_bh_collide(BodyArrays A, DevCtl *ctl, SimSegs seg,
                                                         const unsigned *vals, BhTree t, ull *ev_keys, ll ev_cap)
{
    if (ctl->error) return;
    const ll n = ctl->n;
    const ll M = ctl->bh_count;
    const double rmax = ord_dbl(ctl->bh_rmax);
    int run = -1, root = 0, total = 0;
    float span = 0.f;
    for (ll p = (ll)blockIdx.x * blockDim.x + threadIdx.x; p < M; p += (ll)gridDim.x * blockDim.x) {
        const int r = bh_run_of(t, seg.nsims, p);
        if (r != run) {
            double cx0, cy0, cz0, half0;
            bh_root(t, r, cx0, cy0, cz0, half0);
            /* every coordinate, centre and half in the tree is at most this large */
            span = (float)((fabs(cx0) + fabs(cy0) + fabs(cz0) + 3 * half0) * (1.0 + 0x1p-20));
            root = (int)t.sroot[r];
            total = (int)t.sroot[r + 1];
            run = r;
        }
        const unsigned i = vals[p];
        const unsigned fi = A.flags[i];
        if (fi & NBG_F_COLLIDED) continue; /* Collided's guard (always clear here) */
        const double xi = A.x[i], yi = A.y[i], zi = A.z[i], ri = A.rad[i];
        const unsigned bi = NBG_BEHAVIOR(fi);
        /* The cube test runs in FP32 and only prunes: a node is skipped when
         * its cube lies farther than r_i + r_max plus a bound on every FP32
         * rounding of the coordinates, centres, halves and the test itself
         * (2^-18 of the tree's span); the pairs that remain get the exact
         * FP64 test. */
        const double Rd = ri + rmax;
        if (!(Rd >= 0)) continue; /* a NaN radius collides with nothing */
        const float R = (float)(Rd * (1.0 + 0x1p-20)) + span * 0x1p-18f;
        const float R2 = R * R * (1.0f + 0x1p-18f);
        const float xf = (float)xi, yf = (float)yi, zf = (float)zi;
        /* A leaf is the node whose subtree ends at the next one, so a visit is
         * two loads side by side.  Bound by their latency: with the flags read
         * after them, and the root cube formed for every body, 94 -> 73 us at
         * 131,072 bodies, 468 -> 369 at 10^6. */
        for (int id = root; id < total;) {
            const float4 q = t.fd[id];
            const int skip = t.skip[id];
            const float ax = fmaxf(fabsf(xf - q.x) - q.w, 0.f);
            const float ay = fmaxf(fabsf(yf - q.y) - q.w, 0.f);
            const float az = fmaxf(fabsf(zf - q.z) - q.w, 0.f);
            const bool near = !(ax * ax + ay * ay + az * az > R2);
            if (near && skip == id + 1)
                for (int qq = t.start[id]; qq < t.end[id]; qq++) {
                    const unsigned j = vals[qq];
                    if (j != i) bh_test_pair(A, ctl, ev_keys, ev_cap, i, xi, yi, zi, ri, bi, j);
                }
            id = near ? id + 1 : skip;
        }
        /* bodies of the collection outside its tree: they sit past every
         * tree body in ascending body order, so the collection's are one run */
        const ll lo_b = seg.off[r], hi_b = seg.off[r + 1];
        ll a = M, b = n;
        while (a < b) {
            const ll mid = (a + b) >> 1;
            if ((ll)vals[mid] < lo_b)
                a = mid + 1;
            else
                b = mid;
        }
        for (ll q = a; q < n && (ll)vals[q] < hi_b; q++)
            bh_test_pair(A, ctl, ev_keys, ev_cap, i, xi, yi, zi, ri, bi, vals[q]);
    }
}

/* ---- host side -------------------------------------------------------------- */

int nbg_bh_alloc(BhTree &t, ll cap, ll node_cap)
{
    nbg_bh_free(t);
    const ll nb = rx_blocks(cap);
    const ll nblk = cap / BH_SCAN_TILE + 2;
    bool ok = true;
#define ALLOC(p, cnt) ok = ok && cudaMalloc((void **)&(p), (size_t)(cnt) * sizeof(*(p))) == cudaSuccess
    ALLOC(t.key[0], cap);
    ALLOC(t.key[1], cap);
    ALLOC(t.val[0], cap);
    ALLOC(t.val[1], cap);
    ALLOC(t.hist, nb * RX_BINS);
    ALLOC(t.digits, BH_RS_PASSES * RX_BINS);
    ALLOC(t.base, cap + 1);
    ALLOC(t.blk, nblk);
    ALLOC(t.mass, node_cap);
    ALLOC(t.mx, node_cap);
    ALLOC(t.my, node_cap);
    ALLOC(t.mz, node_cap);
    ALLOC(t.cx, node_cap);
    ALLOC(t.cy, node_cap);
    ALLOC(t.cz, node_cap);
    ALLOC(t.half, node_cap);
    ALLOC(t.skip, node_cap);
    ALLOC(t.start, node_cap);
    ALLOC(t.end, node_cap);
    ALLOC(t.first, node_cap);
    ALLOC(t.parent, node_cap);
    ALLOC(t.flags, node_cap);
    ALLOC(t.fa, node_cap + NBG_MAX_SIMS); /* a slot per collection's root, used or not */
    ALLOC(t.fb, node_cap + NBG_MAX_SIMS);
    ALLOC(t.rec, 2 * (node_cap + NBG_MAX_SIMS));
    ALLOC(t.shalf, node_cap + NBG_MAX_SIMS);
    ALLOC(t.fc, node_cap + NBG_MAX_SIMS);
    ALLOC(t.fd, node_cap);
    ALLOC(t.cbase, node_cap);
    ALLOC(t.ccount, node_cap);
    ALLOC(t.slot, node_cap);
    ALLOC(t.sbox, 6 * (ll)NBG_MAX_SIMS);
    ALLOC(t.scount, NBG_MAX_SIMS + 1);
    ALLOC(t.stree, NBG_MAX_SIMS + 1);
    ALLOC(t.sroot, NBG_MAX_SIMS + 1);
    ALLOC(t.sgrp, NBG_MAX_SIMS + 1);
    ALLOC(t.sunit, NBG_MAX_SIMS + 1);
#undef ALLOC
    if (!ok) {
        nbg_bh_free(t);
        return NBG_E_CUDA;
    }
    t.node_cap = node_cap;
    return NBG_OK;
}

void nbg_bh_free(BhTree &t)
{
    void *ps[] = {t.key[0], t.key[1], t.val[0], t.val[1], t.hist, t.digits, t.base, t.blk, t.mass, t.mx, t.my,
                  t.mz, t.cx, t.cy, t.cz, t.half, t.skip, t.start,
                  t.end, t.first, t.parent, t.flags, t.fa, t.fb, t.rec, t.shalf, t.fc, t.fd, t.cbase, t.ccount, t.slot,
                  t.sbox, t.scount, t.stree, t.sroot, t.sgrp, t.sunit};
    for (void *p : ps) cudaFree(p);
    memset(&t, 0, sizeof t);
}

/* The force and collision pass of one cycle (the replacement of the pair
 * kernel): bounds, keys, sort, nodes, masses, forces (FP64, or the mixed
 * walk), suns, collisions. */
void nbg_launch_bh(const CycleBufs &cb, DevCtl *ctl, cudaStream_t st, bool mixed)
{
    const BhTree &t = cb.t;
    const SimSegs &seg = cb.seg;
    const ll cap = cb.cap;
    const ll gmost = (ll)(cb.sms > 0 ? cb.sms : 1) * 8;
    int g = (int)((cap + BH_BLOCK - 1) / BH_BLOCK < gmost ? (cap + BH_BLOCK - 1) / BH_BLOCK : gmost);
    if (g < 1) g = 1;
    k_bh_reset<<<1, 1024, 0, st>>>(ctl, seg, t);
    k_bh_bounds<<<g, BH_BLOCK, 0, st>>>(cb.a, ctl, seg, t);
    k_bh_segs<<<1, 32, 0, st>>>(ctl, seg, t);
    k_bh_keys<<<g, BH_BLOCK, 0, st>>>(cb.a, ctl, seg, t, t.key[0], t.val[0]);
    const int nb = (int)rx_blocks(cap);
    /* eight passes of the key, then (several collections) two of the
     * collection index: an even count, so the sorted keys and values end in
     * buffer 0 */
    const int passes = seg.nsims > 1 ? BH_RS_PASSES : 8, wide = rx_wide(cap);
    int in = 0;
    for (int pass = 0; pass < passes; pass++) {
        const int shift = pass < 8 ? 8 * pass : 0, simpass = pass < 8 ? -1 : pass - 8;
        unsigned *digits = t.digits + pass * RX_BINS;
        k_bh_rs_hist<<<nb, RX_BLOCK, 0, st>>>(ctl, seg, t.key[in], t.val[in], shift, simpass, wide, t.hist, digits);
        if (wide) k_bh_rs_scan<<<RX_BINS / RX_WARPS, RX_BLOCK, 0, st>>>(ctl, t.hist, digits);
        k_bh_rs_scatter<<<nb, RX_BLOCK, 0, st>>>(ctl, seg, t.key[in], t.val[in], t.key[in ^ 1], t.val[in ^ 1],
                                                   shift, simpass, wide, t.hist, digits);
        in ^= 1;
    }
    const int sb = (int)(cap / BH_SCAN_TILE + 1);
    k_bh_count<<<sb, BH_SCAN_BLOCK, 0, st>>>(ctl, seg, t, t.key[0], t.base, t.blk);
    k_bh_count_top<<<1, 1024, 0, st>>>(ctl, t.blk, t.node_cap);
    k_bh_count_scan<<<sb, BH_SCAN_BLOCK, 0, st>>>(ctl, t.base, t.blk);
    k_bh_roots<<<1, 1024, 0, st>>>(ctl, seg, t, t.base);
    k_bh_nodes<<<g, BH_BLOCK, 0, st>>>(ctl, seg, t.key[0], t.base, t);
    int ng = (int)((t.node_cap + BH_BLOCK - 1) / BH_BLOCK < gmost ? (t.node_cap + BH_BLOCK - 1) / BH_BLOCK : gmost);
    if (ng < 1) ng = 1;
    k_bh_children<<<ng, BH_BLOCK, 0, st>>>(ctl, seg, t);
    k_bh_mass<<<ng, BH_BLOCK, 0, st>>>(cb.a, ctl, t.val[0], t);
    if (mixed) {
        k_bh_prep_mixed<<<ng, BH_BLOCK, 0, st>>>(cb.a, ctl, seg, t);
        /* one wave of resident CTAs, which share the queue of units; 4 CTAs
         * per SM (121 registers, no spill) measured fastest, 2.38 ms for the
         * tree pass of 131,072 Plummer bodies against 2.52 with 5 or 6 */
        const int minb = cb.bh_shape == 1 ? 5 : cb.bh_shape == 2 ? 6 : 4;
        const ll wgroups = cap / 32 + 1 + seg.nsims;
        const int gw = (int)(wgroups < (ll)cb.sms * minb ? wgroups : (ll)cb.sms * minb);
        switch (cb.bh_shape) {
        case 1: k_bh_force_mixed<5><<<gw, BHW_BLOCK, 0, st>>>(cb.a, ctl, seg, t.val[0], t); break;
        case 2: k_bh_force_mixed<6><<<gw, BHW_BLOCK, 0, st>>>(cb.a, ctl, seg, t.val[0], t); break;
        default: k_bh_force_mixed<4><<<gw, BHW_BLOCK, 0, st>>>(cb.a, ctl, seg, t.val[0], t); break;
        }
    } else {
        k_bh_prep64<<<ng, BH_BLOCK, 0, st>>>(cb.a, ctl, t);
        const ll wgroups = cap / 32 + 1 + seg.nsims;
        const int gw = (int)(wgroups < (ll)cb.sms * 5 ? wgroups : (ll)cb.sms * 5);
        k_bh_force<<<gw, BHW_BLOCK, 0, st>>>(cb.a, ctl, seg, t.val[0], t);
    }
    k_bh_sun<<<64, BH_BLOCK, 0, st>>>(cb.a, ctl, seg);
    k_bh_collide<<<g, BH_BLOCK, 0, st>>>(cb.a, ctl, seg, t.val[0], t, cb.ev_keys, cb.ev_cap);
}

int nbg_bh_launches(const CycleBufs &cb, bool mixed)
{
    const int passes = cb.seg.nsims > 1 ? BH_RS_PASSES : 8;
    /* reset, bounds, segs, keys; the sort; count, top, scan, roots, nodes;
     * children, masses; prep, walk; suns, collisions */
    return 4 + (2 + rx_wide(cb.cap)) * passes + 5 + 2 + 2 + 2;
}
