// Host comparison of nbg_exact.h with the host's sqrt, product and division
// (IEEE 754, correctly rounded): random operands over the whole accepted range, operands
// whose significands are at the ends of their range, and roots and quotients
// built to lie as near a rounding boundary as 53-bit operands allow.  The
// FP32 seed is moved by up to two units, which covers the device's
// approximation (2^-22.9 relative).
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstdint>

static int g_seed_off = 0;
#define NBX_SEED_OFF g_seed_off
#include "nbg_exact.h"

static uint64_t g_state = 88172645463325252ull;
static uint64_t rnd()
{
    g_state ^= g_state << 13;
    g_state ^= g_state >> 7;
    g_state ^= g_state << 17;
    return g_state * 0x2545f4914f6cdd1dull;
}
static double make(uint32_t e, uint64_t frac) { return nbx_double(((uint64_t)e << 52) | (frac & NBX_FRAC)); }
static uint64_t edge()
{
    switch (rnd() % 6) {
    case 0: return rnd() % 4;
    case 1: return NBX_FRAC - rnd() % 4;
    case 2: return (1ull << (rnd() % 52)) - rnd() % 2;
    case 3: return NBX_FRAC << (rnd() % 52);
    case 4: return 0x6a09e667f3bccull + rnd() % 5 - 2; // near sqrt(2)
    default: return rnd();
    }
}
static long long bad = 0, checked = 0;

// a number with exponent field 1023 +- span, or zero now and then
static double num(uint32_t span, bool edges)
{
    const double v = make(1023 - span + (uint32_t)(rnd() % (2 * span + 1)), edges ? edge() : rnd());
    return rnd() & 1 ? v : -v;
}
static void same(const char *what, double want, uint64_t got, double a, double b)
{
    checked++;
    if (nbx_bits(want) != got && bad++ < 8) printf("%s %a, %a: want %a got %a\n", what, a, b, want, nbx_double(got));
}

// the whole term of a pair: s, gm = g m, d
static void one(double s, double g, double m, const double d[3])
{
    const uint64_t sb = nbx_bits(s);
    if (!nbx_root_ok(sb) || !nbx_mass_ok(nbx_bits(g)) || !nbx_mass_ok(nbx_bits(m))) return;
    const nbx_root root = nbx_sqrt(sb);
    const nbx_div r = root.r;
    const double dist = sqrt(s), gm = g * m;
    same("sqrt", dist, nbx_div_bits(r), s, 0);
    const double d2 = dist * dist, f = gm / d2;
    same("force over the operand", gm / s,
         nbx_pack(nbx_quot(nbx_mul(nbx_unpack(nbx_bits(g)), nbx_unpack(nbx_bits(m))), nbx_operand(root))), gm, s);
    if (!nbx_square_ok(root)) return;
    const nbx_div r2 = nbx_square(root);
    same("square", d2, nbx_div_bits(r2), dist, dist);
    const nbx_num xg = nbx_mul(nbx_unpack(nbx_bits(g)), nbx_unpack(nbx_bits(m)));
    same("mass product", gm, nbx_pack(xg), g, m);
    const nbx_num xf = nbx_quot(xg, r2);
    same("force", f, nbx_pack(xf), gm, d2);
    for (int c = 0; c < 3; c++) {
        if (d[c] == 0 || !nbx_diff_ok(nbx_bits(d[c]))) continue;
        const nbx_num xd = nbx_unpack(nbx_bits(d[c]));
        same("difference squared", d[c] * d[c], nbx_pack(nbx_mul(xd, xd)), d[c], d[c]);
        const nbx_num xa = nbx_mul(xf, xd);
        const double a = f * d[c];
        same("product", a, nbx_pack(xa), f, d[c]);
        same("term", a / dist, nbx_pack(nbx_quot(xa, r)), a, dist);
    }
}

int main(int argc, char **argv)
{
    const long long n = argc > 1 ? atoll(argv[1]) : 3000000;
    if (argc > 2) g_state ^= (uint64_t)atoll(argv[2]) << 20;
    for (long long k = 0; k < n; k++) {
        g_seed_off = (int)(rnd() % 5) - 2;
        double d[3];
        const uint32_t span = k % 4 ? 40 : 150;
        for (double &v : d) v = rnd() % 64 == 0 ? 0.0 : num(span, k % 3 == 0);
        double s = d[0] * d[0] + d[1] * d[1] + d[2] * d[2];
        if (k % 5 == 1) s = make(1023 - 302 + (uint32_t)(rnd() % 605), edge());
        if (k % 5 == 2) {
            // s within a unit or two of the square of a 54-bit number: the
            // root near a rounding boundary
            const uint64_t h = (1ull << 53) | (rnd() & ((1ull << 53) - 1));
            uint64_t top = (uint64_t)(((unsigned __int128)h * h) >> 54);
            while (top >> 53) top >>= 1;
            s = make(1000 + (uint32_t)(rnd() % 47), top + rnd() % 3 - 1);
        }
        if (k % 11 == 4) {
            // roots with few bits: ties of their squares' rounding
            const double q = make(1000 + (uint32_t)(rnd() % 47), (rnd() & 0x7ffffffull) << 25);
            s = q * q;
            if (rnd() & 1) s = nbx_double(nbx_bits(s) + rnd() % 3 - 1);
        }
        double g = num(200, k % 2 == 0), m = num(200, k % 7 == 0);
        if (k % 7 == 3) {
            // g m within a unit of (q + 1/2) d2: the quotient near a boundary
            const double dist = sqrt(s), d2 = dist * dist;
            const uint64_t B = (nbx_bits(d2) & NBX_FRAC) | NBX_ONE, Q = (rnd() & NBX_FRAC) | NBX_ONE;
            uint64_t top = (uint64_t)(((unsigned __int128)B * (2 * Q + 1)) >> 53);
            while (top >> 53) top >>= 1;
            g = make(1023 + (uint32_t)(rnd() % 40), top + rnd() % 3 - 1);
            m = 1.0;
        }
        if (k % 7 == 5) {
            // products with few bits: ties of the rounding
            g = make(1023, (rnd() & 0x7ffffffull) << 25);
            m = make(1023, (rnd() & 0x7ffffffull) << 25);
            d[0] = make(1023, (rnd() & 0x7ffffffull) << 25);
        }
        one(s, g, m, d);
    }
    printf("checked %lld, bad %lld\n", checked, bad);
    return bad != 0;
}
