/*
 * nbg_radix.cuh - one pass of a stable LSD radix sort (8-bit digits) over keys
 * with 32-bit values, as device functions for the kernels that sort: the spatial
 * order (k_sort.cu) and the Barnes-Hut keys (k_bh.cu).
 *
 * A pass is a histogram of each block's RX_TILE keys, with the digits' totals,
 * which all blocks add to (zeroed before), and a scatter.  Up to RX_NARROW
 * blocks, the histogram lies block by block and each block of the scatter adds
 * up the rows of those before it; past that ("wide"), the sum would grow with
 * the square of the blocks, and a scan between the two turns the histogram,
 * digit by digit, into offsets.  Small tiles, so 131,072 keys make 128
 * blocks, and no barrier between a block's keys; a warp ranks its consecutive
 * keys with match masks, in order.
 */
#ifndef NBG_RADIX_CUH
#define NBG_RADIX_CUH

#include "nbg_internal.cuh"

#define RX_BLOCK 256
#define RX_WARPS (RX_BLOCK / 32)
#define RX_ITEMS 4
#define RX_TILE (RX_BLOCK * RX_ITEMS)
#define RX_BINS 256
/* most blocks whose scatter sums the histogram itself: the rows come one after
 * another from the L2 (50,001 keys, 49 blocks: 13.1 us, against 3.5 for the scan
 * and 4.7 for a scatter without them) */
#define RX_NARROW 32
static_assert(RX_BLOCK == RX_BINS, "a thread per digit");

static inline ll rx_blocks(ll n) { return (n + RX_TILE - 1) / RX_TILE; }
static inline int rx_wide(ll cap) { return rx_blocks(cap) > RX_NARROW; }

/* digit(k): of the key at position k */
template <class DIGIT>
__device__ __forceinline__ void rx_hist(ll n, int wide, unsigned *hist, unsigned *digits, DIGIT digit)
{
    __shared__ unsigned cnt[RX_BINS];
    const ll nb = (n + RX_TILE - 1) / RX_TILE, b = blockIdx.x;
    if (b >= nb) return;
    const int tid = threadIdx.x;
    cnt[tid] = 0;
    __syncthreads();
#pragma unroll
    for (int q = 0; q < RX_ITEMS; q++) {
        const ll k = b * RX_TILE + (ll)q * RX_BLOCK + tid;
        if (k < n) atomicAdd(&cnt[digit(k)], 1u);
    }
    __syncthreads();
    const unsigned c = cnt[tid];
    hist[wide ? (ll)tid * nb + b : b * RX_BINS + tid] = c;
    if (c) atomicAdd(&digits[tid], c);
}

/* thread d: the elements of the digits below d */
__device__ __forceinline__ unsigned rx_digit_start(const unsigned *digits, unsigned *wtot)
{
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const unsigned v = digits[threadIdx.x];
    unsigned x = v;
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) wtot[w] = x;
    __syncthreads();
    for (int u = 0; u < w; u++) x += wtot[u];
    return x - v;
}

/* a warp to a digit's row of the histogram; RX_BINS / RX_WARPS blocks */
__device__ __forceinline__ void rx_scan(ll n, unsigned *hist, const unsigned *digits)
{
    __shared__ unsigned wtot[RX_WARPS], start[RX_BINS];
    const ll nb = (n + RX_TILE - 1) / RX_TILE;
    const int lane = threadIdx.x & 31, d = blockIdx.x * RX_WARPS + (threadIdx.x >> 5);
    start[threadIdx.x] = rx_digit_start(digits, wtot);
    __syncthreads();
    unsigned carry = start[d];
    unsigned *row = hist + (ll)d * nb;
    for (ll c = 0; c < nb; c += 32) {
        const unsigned v = c + lane < nb ? row[c + lane] : 0u;
        unsigned x = v;
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        if (c + lane < nb) row[c + lane] = carry + x - v;
        carry += __shfl_sync(0xffffffffu, x, 31);
    }
}

/* digit(key, val) */
template <class K, class DIGIT>
__device__ __forceinline__ void rx_scatter(ll n, int wide, const K *keys_in, const unsigned *vals_in, K *keys_out,
                                           unsigned *vals_out, const unsigned *hist, const unsigned *digits,
                                           DIGIT digit)
{
    __shared__ unsigned wtot[RX_WARPS], cnt[RX_WARPS][RX_BINS];
    const ll nb = (n + RX_TILE - 1) / RX_TILE, b = blockIdx.x;
    if (b >= nb) return;
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const unsigned lt = (1u << lane) - 1u;
    /* a warp's keys are consecutive: its first, then 32 at a time */
    const ll k0 = b * RX_TILE + (ll)w * (32 * RX_ITEMS) + lane;
    K key[RX_ITEMS];
    unsigned val[RX_ITEMS], rank[RX_ITEMS], dig[RX_ITEMS];
#pragma unroll
    for (int q = 0; q < RX_ITEMS; q++) {
        const bool ok = k0 + 32 * q < n;
        key[q] = ok ? keys_in[k0 + 32 * q] : (K)0;
        val[q] = ok ? vals_in[k0 + 32 * q] : 0u;
    }
    /* where the block's elements of digit tid start */
    unsigned at;
    if (wide) {
        at = hist[(ll)tid * nb + b];
    } else {
        at = rx_digit_start(digits, wtot);
        const unsigned *h = hist + tid;
#pragma unroll 8
        for (int u = 0; u < (int)b; u++) at += h[u * RX_BINS];
    }
    for (int c = tid; c < RX_BINS * RX_WARPS; c += RX_BLOCK) (&cnt[0][0])[c] = 0;
    __syncthreads();
#pragma unroll
    for (int q = 0; q < RX_ITEMS; q++) {
        const bool ok = k0 + 32 * q < n;
        const unsigned d = ok ? digit(key[q], val[q]) : RX_BINS; /* never matches a real digit */
        const unsigned peers = __match_any_sync(0xffffffffu, d);
        const unsigned before = __popc(peers & lt);
        const unsigned old = ok ? cnt[w][d] : 0u;
        dig[q] = d;
        rank[q] = old + before;
        __syncwarp();
        if (ok && before == 0) cnt[w][d] = old + __popc(peers);
        __syncwarp();
    }
    __syncthreads();
    for (int u = 0; u < RX_WARPS; u++) {
        const unsigned c = cnt[u][tid];
        cnt[u][tid] = at;
        at += c;
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < RX_ITEMS; q++)
        if (k0 + 32 * q < n) {
            const unsigned pos = cnt[w][dig[q]] + rank[q];
            keys_out[pos] = key[q];
            vals_out[pos] = val[q];
        }
}

#endif /* NBG_RADIX_CUH */
