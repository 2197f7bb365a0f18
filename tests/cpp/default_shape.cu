// The mixed kernel's shape by default (nbg_internal.cuh): symmetric where every
// collection is large and the j partials take at most an eighth of the memory.
#include <cstdio>

#include "nbg_internal.cuh"

int main()
{
    int bad = 0;
    const unsigned long long gb = 1ull << 30, big = 280 * gb;
    const ll m = 98304, k = NBG_MIX_SYM_MIN_N;
    auto want = [&](int nsims, const ll *c, unsigned long long bytes, int v) {
        if (nbg_default_shape(nsims, c, bytes) != v) {
            printf("%d collections, the first of %lld bodies: %d, not %d\n", nsims, (long long)c[0],
                   nbg_default_shape(nsims, c, bytes), v);
            bad++;
        }
    };
    const ll none[] = {0}, one[] = {1}, few[] = {NBG_MIX_FEW_N - 1}, more[] = {NBG_MIX_FEW_N};
    want(1, none, big, NBG_MIX_ONE_SIDED_FEW);
    want(1, one, big, NBG_MIX_ONE_SIDED_FEW);
    want(1, few, big, NBG_MIX_ONE_SIDED_FEW);
    want(1, more, big, NBG_MIX_ONE_SIDED);
    const ll below[] = {m - 512}, at[] = {m - 511}, m1[] = {1 << 20}, huge[] = {1ll << 30};
    want(1, below, big, NBG_MIX_ONE_SIDED); // one block less
    want(1, at, big, NBG_MIX_SYM);
    want(1, m1, big, NBG_MIX_SYM);
    want(1, m1, 64 * gb, NBG_MIX_ONE_SIDED); // 16 GB of j partials
    want(1, huge, big, NBG_MIX_ONE_SIDED);
    want(1, at, 0, NBG_MIX_ONE_SIDED); // size unknown
    const ll two[] = {m, k}, mixed[] = {2 * m, 0, 3 * m}, small[] = {2 * m, k - 1};
    want(2, two, big, NBG_MIX_SYM);
    want(3, mixed, big, NBG_MIX_ONE_SIDED);
    want(2, small, big, NBG_MIX_ONE_SIDED);
    // every unit counts: collections that are too few alone, and that fit alone
    static ll some[16], many[64], batch[1000];
    for (ll &c : some) c = k;
    for (ll &c : many) c = 1 << 18;
    for (ll &c : batch) c = NBG_MIX_SYM_MIN_N - 1;
    want(1, some, big, NBG_MIX_ONE_SIDED_FEW);
    want(15, some, big, NBG_MIX_ONE_SIDED_FEW);
    want(16, some, big, NBG_MIX_SYM);
    want(1, many, big, NBG_MIX_SYM);
    want(64, many, big, NBG_MIX_ONE_SIDED);
    want(1000, batch, big, NBG_MIX_ONE_SIDED_FEW);
    printf("default shape bad %d\n", bad);
    return bad != 0;
}
