/*
 * nbg_exact.h - correctly rounded FP64 products, quotients and square roots from
 * integer arithmetic.
 *
 * GB300 runs FP64 at 1/64 of its FP32 rate, and a pair of the plain form
 * needs one square root and four divisions, about ten FP64-pipe operations
 * each when the compiler expands them, and eight products.  Here they run on
 * the integer pipes, on 53-bit significands:
 *
 *   - 1/sqrt from the FP32 approximation and one third-order Newton step in
 *     64-bit fixed point (relative error below 2^-59);
 *   - candidates for sqrt and quotients as products with it, each within
 *     0.52 units in the last place of the exact value;
 *   - the exact remainder, S 2^k - D^2 or A 2^k - Q B, taken modulo 2^64: the
 *     candidate is so close that the low 64 bits determine it;
 *   - a correction by one unit if the remainder says so.
 *
 * A remainder decides the rounding exactly, so the results are those of IEEE
 * 754 round-to-nearest-even for every operand in range: a quotient or square
 * root of 53-bit numbers is never half way between two of them.  (2 R = B
 * would need B to be divisible by 2^53, and a tie of the root would need an
 * odd square to be even.)  Operands out of range (zero, subnormal, infinite,
 * NaN, or so large or small that a result might be) are refused, and the
 * caller takes the ordinary operators for the pair.
 *
 * Written from those definitions; tests/cpp/exact_host.cu compares it with the
 * host's sqrt and division.
 */
#ifndef NBG_EXACT_H
#define NBG_EXACT_H

#include <stdint.h>
#include <string.h>
#if !defined(__CUDA_ARCH__)
#include <math.h>
#endif

#if defined(__CUDACC__)
#define NBG_XFN __host__ __device__ __forceinline__
#else
#define NBG_XFN static inline
#endif

NBG_XFN uint64_t nbx_bits(double v)
{
#if defined(__CUDA_ARCH__)
    return (uint64_t)__double_as_longlong(v);
#else
    uint64_t b;
    memcpy(&b, &v, 8);
    return b;
#endif
}

NBG_XFN double nbx_double(uint64_t b)
{
#if defined(__CUDA_ARCH__)
    return __longlong_as_double((long long)b);
#else
    double v;
    memcpy(&v, &b, 8);
    return v;
#endif
}

NBG_XFN uint64_t nbx_mulhi(uint64_t a, uint64_t b)
{
#if defined(__CUDA_ARCH__)
    return __umul64hi(a, b);
#else
    return (uint64_t)(((unsigned __int128)a * b) >> 64);
#endif
}

/* bits of an FP32 approximation of 1/sqrt of the float with bits b, which is
 * in [1, 4); relative error below 2^-22 */
NBG_XFN uint32_t nbx_rsqrt_seed(uint32_t b)
{
#if defined(__CUDA_ARCH__)
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(__uint_as_float(b)));
    return __float_as_uint(y);
#else
#ifndef NBX_SEED_OFF
#define NBX_SEED_OFF 0
#endif
    float x, y;
    memcpy(&x, &b, 4);
    y = (float)(1.0 / sqrt((double)x));
    uint32_t r;
    memcpy(&r, &y, 4);
    return r + NBX_SEED_OFF; /* the host test moves the seed by a unit or two */
#endif
}

/* Operands taken: of a root, 2^-302 .. 2^302; of a coordinate difference,
 * 2^-150 .. 2^150; of a mass, 2^-200 .. 2^200.  Every product, quotient and
 * root of a pair term is then a normal number, below 2^1000 and above
 * 2^-1000.  (A squared distance is within its range when its differences are
 * zero or in theirs, and not all zero.) */
NBG_XFN int nbx_within(uint64_t bits, uint32_t span)
{
    return ((uint32_t)(bits >> 52) & 0x7ffu) - (1023u - span) <= 2u * span;
}
NBG_XFN int nbx_root_ok(uint64_t bits) { return !(bits >> 63) && nbx_within(bits, 302); }
/* +-0, from the words: asked of the 64-bit pattern the compiler makes it a
 * comparison on the FP64 pipe */
NBG_XFN int nbx_zero(uint64_t bits) { return (((uint32_t)(bits >> 32) << 1) | (uint32_t)bits) == 0; }
NBG_XFN int nbx_diff_ok(uint64_t bits) { return nbx_within(bits, 150) || nbx_zero(bits); }
NBG_XFN int nbx_mass_ok(uint64_t bits) { return nbx_within(bits, 200); }

#define NBX_ONE 0x10000000000000ull /* 2^52 */
#define NBX_FRAC 0xfffffffffffffull

/* A number: its significand a in [2^52, 2^53) and e = sign << 11 | exponent
 * field. */
struct nbx_num {
    uint64_t a;
    uint32_t e;
};
NBG_XFN nbx_num nbx_unpack(uint64_t bits)
{
    nbx_num n;
    n.a = (bits & NBX_FRAC) | NBX_ONE;
    n.e = (uint32_t)(bits >> 52);
    return n;
}
NBG_XFN uint64_t nbx_pack(const nbx_num &n) { return ((uint64_t)n.e << 52) + (n.a - NBX_ONE); }

/* v 2^(32 + sh) mod 2^64, sh < 32 */
NBG_XFN uint64_t nbx_top(uint64_t v, uint32_t sh) { return (uint64_t)((uint32_t)v << sh) << 32; }

/* RN of the product of two significands, as a significand; up says whether
 * it is that of a product in [2, 4).  The top 64 bits of the 106-bit product
 * and whether any bit below them is set decide the rounding. */
NBG_XFN uint64_t nbx_mul_sig(uint64_t a, uint64_t b, uint32_t &up)
{
    uint64_t hi = nbx_mulhi(a << 11, b << 11);
    up = (uint32_t)(hi >> 63);
    hi = (hi << (up ^ 1u)) | (((a * b) << 22) != 0 ? 1u : 0u); /* the significand's 53 bits on top */
    uint64_t q = hi >> 11;
    q += ((uint32_t)hi & 2047u) + ((uint32_t)q & 1u) > 1024u ? 1u : 0u;
    const uint32_t c = (uint32_t)(q >> 53); /* rounded up to the next power of two */
    up += c;
    return q >> c;
}

/* RN(x y), for operands whose product is normal */
NBG_XFN nbx_num nbx_mul(const nbx_num &x, const nbx_num &y)
{
    nbx_num r;
    uint32_t up;
    r.a = nbx_mul_sig(x.a, y.a, up);
    r.e = ((x.e ^ y.e) & 0x800u) | ((x.e & 0x7ffu) + (y.e & 0x7ffu) + up - 1023u);
    return r;
}

/* A divisor: its significand d in [2^52, 2^53), exponent field e, and
 * y = 2^115 / d within 2^-58 of itself (2^62 < y <= 2^63). */
struct nbx_div {
    uint64_t d, y;
    int e;
};

/* A root with what its square needs: its operand's significand S (times
 * 2^odd) and the exact remainder, d^2 = S 2^(52 + odd) - rem. */
struct nbx_root {
    nbx_div r;
    uint64_t S, y1; /* y1 = 2^63 / sqrt(S 2^odd / 2^52) within 2^-59 */
    int64_t rem;
    uint32_t odd;
    int e; /* the operand's exponent field */
};

/* RN(sqrt(s)) as a divisor, for s_bits in range.  Its value is
 * nbx_double(nbx_div_bits(root.r)). */
NBG_XFN nbx_root nbx_sqrt(uint64_t s_bits)
{
    const uint32_t ef = (uint32_t)(s_bits >> 52);
    const uint32_t odd = (ef & 1u) ^ 1u; /* s = m 2^(2 k), m = f in [1, 2) or 2 f in [2, 4) */
    const uint64_t S = (s_bits & NBX_FRAC) | NBX_ONE;
    const uint64_t m = S << (9 + odd); /* m 2^61 */
    uint32_t yb = nbx_rsqrt_seed(((127u + odd) << 23) | ((uint32_t)(S >> 29) & 0x7fffffu));
    yb = yb < 0x3f000000u ? 0x3f000000u : yb; /* the exact value is in (1/2, 1] */
    yb = yb > 0x3f800000u ? 0x3f800000u : yb;
    const uint32_t y0 = ((yb & 0x7fffffu) | 0x800000u) << ((yb >> 23) - 126u); /* y 2^24, y in (1/2, 1] */
    /* e0 = 1 - m y0^2 (scale 2^60), below 2^-20 */
    const int64_t e0 = (int64_t)((1ull << 60) - nbx_mulhi(m, ((uint64_t)y0 * y0) << 15));
    /* y1 = y0 (1 + e0 / 2 + 3/8 e0^2): the next term is below 2^-61 */
    const int32_t eh = (int32_t)(e0 >> 20);
    const int32_t e2 = (int32_t)(((int64_t)eh * eh) >> 16);
    const int64_t c = e0 + ((e2 * 3) >> 6);                                     /* scale 2^61 */
    const uint64_t y1 = ((uint64_t)y0 << 39) + (uint64_t)(((int64_t)y0 * c) >> 22); /* scale 2^63 */
    nbx_root v;
    uint64_t d = (nbx_mulhi(m, y1) + 128u) >> 8;
    int64_t rem = (int64_t)(nbx_top(S, 20 + odd) - d * d); /* S 2^(52 + odd) - d^2 */
    if (rem > (int64_t)d) {
        rem -= (int64_t)(2 * d + 1);
        d += 1;
    } else if (rem <= -(int64_t)d) {
        rem += (int64_t)(2 * d - 1);
        d -= 1;
    }
    /* y1 is 1 / sqrt(m); the divisor is the rounded root, sqrt(m) less
     * rem / (2 d): y1 (1 + rem / (2 d^2)) */
    const int32_t y8 = (int32_t)(y0 >> 16);
    v.r.d = d;
    v.r.y = y1 + (uint64_t)(((int64_t)(int32_t)(rem >> 22) * (y8 * y8 * y8)) >> 44);
    v.r.e = (int)((ef + 1023u - odd) >> 1);
    v.S = S;
    v.y1 = y1;
    v.rem = rem;
    v.odd = odd;
    v.e = (int)ef;
    return v;
}

NBG_XFN uint64_t nbx_div_bits(const nbx_div &r) { return ((uint64_t)(uint32_t)r.e << 52) + (r.d - NBX_ONE); }

/* RN(d d) of a root d as a divisor: 1 / (d d) adjusted to the rounded square.
 * The square is S 2^(52 + odd) - rem with |rem| <= d, so it rounds to S or a
 * neighbour of S; the tie, possible for odd, goes to the even one.  Not for an
 * S at either end of its range, whose neighbour may have another exponent. */
NBG_XFN int nbx_square_ok(const nbx_root &v)
{
    return v.S - (NBX_ONE + 1) <= NBX_FRAC - 2; /* 2^52 < S < 2^53 - 1 */
}
NBG_XFN nbx_div nbx_square(const nbx_root &v)
{
    nbx_div q;
    const int64_t half = (int64_t)(1ull << (51 + v.odd));
    const int64_t tie = (int64_t)(v.S & 1u); /* an odd S gives way at a tie */
    int64_t diff = -v.rem;
    uint64_t d = v.S;
    if (diff > half - tie) {
        d += 1;
        diff -= 2 * half;
    } else if (diff < tie - half) {
        d -= 1;
        diff += 2 * half;
    }
    q.d = d;
    q.e = 2 * v.r.e - 1023 + (int)v.odd;
    const uint64_t y = nbx_mulhi(v.r.y, v.r.y) << (1 + v.odd);
    const int32_t y8 = (int32_t)(y >> 55);
    q.y = y + (uint64_t)(((int64_t)(int32_t)(diff >> (21 + v.odd)) * (y8 * y8)) >> 36);
    return q;
}

/* The operand of a root itself as a divisor. */
NBG_XFN nbx_div nbx_operand(const nbx_root &v)
{
    nbx_div q;
    q.d = v.S;
    q.e = v.e;
    q.y = nbx_mulhi(v.y1, v.y1) << (1 + v.odd);
    return q;
}

/* RN(n / r) */
NBG_XFN nbx_num nbx_quot(const nbx_num &n, const nbx_div &r)
{
    nbx_num v;
    const uint32_t lt = n.a < r.d ? 1u : 0u; /* the quotient of the significands in [1/2, 1) or [1, 2) */
    const uint64_t w = nbx_mulhi(n.a << 11, r.y); /* a 2^62 / d */
    uint64_t q = ((w << lt) + 512u) >> 10;
    const int64_t R = (int64_t)(nbx_top(n.a, 20 + lt) - q * r.d); /* a 2^(52 + lt) - q d */
    const int64_t h = 2 * R;
    q += h > (int64_t)r.d ? 1u : 0u;
    q -= h < -(int64_t)r.d ? 1u : 0u;
    v.a = q;
    v.e = n.e + 1023u - lt - (uint32_t)r.e;
    return v;
}

#endif /* NBG_EXACT_H */
