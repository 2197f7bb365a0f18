// The grid cell's octant path against the descent's (nbg_octant.h): random points,
// points on and next to the faces that the descent compares with, cubes on and
// far off the origin, small and large.
#include <cmath>
#include <cstdint>
#include <cstdio>

#include "nbg_octant.h"

static uint64_t s = 0x9e3779b97f4a7c15ull;
static uint64_t rnd()
{
    s ^= s << 13;
    s ^= s >> 7;
    s ^= s << 17;
    return s;
}
static double unit() { return (double)(rnd() >> 11) * 0x1p-53; }

int main()
{
    long long bad = 0, sure = 0, all = 0, random_sure = 0, random_all = 0;
    const double halves[] = {1.0, 67.2, 1e-3, 3.7e11, 1e-30, 1e60, 1e-240, 1e240, 1e-260, 1e260, 0.0, INFINITY, NAN};
    const double offs[] = {0.0, 1e-3, 1.0, -37.0, 1e3, -5e5, 9e5, 2e6, 1e9, 1e15};
    for (double half : halves)
        for (double off : offs) {
            const double c[3] = {off * half, -0.7 * off * half, (0.3 * off + 0.1) * half};
            const NbgOctGrid g = nbg_oct_grid(c[0], c[1], c[2], half);
            for (int n = 0; n < 20000; n++) {
                double p[3];
                const int kind = n % 4;
                for (int a = 0; a < 3; a++) {
                    if (kind == 0) {
                        p[a] = c[a] + half * (2.0 * unit() - 1.0);
                    } else {
                        // a centre of the descent, at a random depth
                        double v = c[a], h = half;
                        for (int d = (int)(rnd() % 21); d > 0; d--) {
                            v = (rnd() & 1) ? v + h / 2 : v - h / 2;
                            h /= 2;
                        }
                        // on it, some units in the last place off, or some 2^-30 of a cell off
                        if (kind == 2)
                            for (int q = (int)(rnd() % 4); q > 0; q--) v = nextafter(v, (rnd() & 1) ? INFINITY : -INFINITY);
                        if (kind == 3) v += half * 0x1p-50 * (double)(int)(rnd() % 2001 - 1000);
                        p[a] = v;
                    }
                }
                if (n % 97 == 0) p[n % 3] = n % 2 ? NAN : c[n % 3] + 1.5 * half;
                unsigned long long key = 0;
                const int ok = nbg_oct_cell(g, p[0], p[1], p[2], key);
                all++;
                sure += ok;
                if (kind == 0 && fabs(off) <= 1e3 && half >= 1e-240 && half <= 1e240) {
                    random_all++;
                    random_sure += ok;
                }
                if (ok && key != nbg_oct_path(p[0], p[1], p[2], c[0], c[1], c[2], half)) bad++;
            }
        }
    printf("octant bad %lld, sure %lld of %lld, of random points %lld of %lld\n", bad, sure, all, random_sure, random_all);
    return bad != 0 || random_sure * 100 < random_all * 95;
}
