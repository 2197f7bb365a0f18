// Host checks of two rules of the mixed pair pass (nbg_internal.cuh).
//  - nbg_hilbert: for every cube up to 2^7 a side, a bijection whose
//    neighbours on the curve are neighbours in the cube;
//  - the chunk cut at its finest, 32 units a chunk (one-sided) and 4
//    (symmetric): every chunk holds work and every unit maps to its chunk.
#include <cstdio>
#include <cstdlib>
#include <vector>

#include "nbg_internal.cuh"

static long long hilbert_bad()
{
    long long bad = 0;
    for (int b = 1; b <= 7; b++) {
        const int m = 1 << b;
        std::vector<int> at((size_t)m * m * m, -1);
        for (int x = 0; x < m; x++)
            for (int y = 0; y < m; y++)
                for (int z = 0; z < m; z++) {
                    const unsigned k = nbg_hilbert(x, y, z, b);
                    if (k >= at.size() || at[k] != -1) {
                        bad++;
                        continue;
                    }
                    at[k] = (x * m + y) * m + z;
                }
        for (size_t k = 1; k < at.size(); k++) {
            const int p = at[k - 1], q = at[k];
            const int d = abs(p / m / m - q / m / m) + abs(p / m % m - q / m % m) + abs(p % m - q % m);
            if (p < 0 || q < 0 || d != 1) bad++;
        }
    }
    // 10 bits (the single-collection grid): one key per cell along a diagonal
    // block, all below 2^30
    std::vector<unsigned> seen;
    for (unsigned x = 500; x < 532; x++)
        for (unsigned y = 1000; y < 1024; y++) {
            const unsigned k = nbg_hilbert(x, y, x ^ y, 10);
            if (k >> 30) bad++;
            for (unsigned s : seen)
                if (s == k) bad++;
            seen.push_back(k);
        }
    return bad;
}

static long long cut_bad(int per)
{
    long long bad = 0;
    const int Cs[] = {1, 2, 3, 4, 5, 7, 10, 33, 100, 608, 4864, 19456};
    for (int C : Cs)
        for (long long extra : {0LL, 1LL, 3LL, (long long)C / 2, (long long)C - 1, 17LL * C + 5}) {
            const ll W = (ll)per * C + extra;
            for (ll c = 0; c < C; c++) {
                const ll a = nbg_chunk_start(c, C, W), b = nbg_chunk_start(c + 1, C, W);
                if (b <= a) bad++;
            }
            if (nbg_chunk_start(0, C, W) != 0 || nbg_chunk_start(C, C, W) != W) bad++;
            for (ll u = 0; u < W; u += W > 100000 ? 7 : 1) {
                const int c = nbg_work_chunk(u, C, W);
                if (c < 0 || c >= C || nbg_chunk_start(c, C, W) > u || nbg_chunk_start(c + 1, C, W) <= u) bad++;
            }
        }
    return bad;
}

int main()
{
    const long long h = hilbert_bad(), c = cut_bad(NBG_MIX_FLOOR_WORK) + cut_bad(4);
    printf("hilbert bad %lld, cut bad %lld\n", h, c);
    return h + c != 0;
}
