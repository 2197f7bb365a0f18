/*
 * nbg_octant.h - the octant path of a point in a root cube, 21 levels of 3 bits
 * (x lowest), as the Barnes-Hut tree sorts bodies by it.
 *
 * nbg_oct_path descends the cube as the reference's tree does (octree.go:
 * comparisons with the cubes' centres, centres moved by half / 2):
 * 170 FP64 operations a body.  nbg_oct_cell has the same bits from the
 * cell of a grid of 2^21 cells a side, 9 FP64 operations, or says that it is not
 * sure: a coordinate within rounding of a cell's face may be on either side of
 * the centre that the descent has there.
 *
 * Plain FP64 without contraction, the same on the host;
 * tests/cpp/octant_host.cu compares the two.
 */
#ifndef NBG_OCTANT_H
#define NBG_OCTANT_H

#include <stdint.h>
#include <string.h>
#include <math.h>

#if defined(__CUDACC__)
#define NBG_OFN __host__ __device__ __forceinline__
#else
#define NBG_OFN static inline
#endif

#define NBG_OCT_LEVELS 21

NBG_OFN unsigned long long nbg_oct_path(double x, double y, double z, double cx, double cy, double cz, double half)
{
    unsigned long long key = 0;
    for (int d = 0; d < NBG_OCT_LEVELS; d++) {
        const unsigned oct = (x >= cx ? 1u : 0u) | (y >= cy ? 2u : 0u) | (z >= cz ? 4u : 0u);
        key = (key << 3) | oct;
        const double q = half / 2;
        cx = (oct & 1u) ? cx + q : cx - q;
        cy = (oct & 2u) ? cy + q : cy - q;
        cz = (oct & 4u) ? cz + q : cz - q;
        half = half / 2;
    }
    return key;
}

/* bit b of v to bit 3 b */
NBG_OFN unsigned long long nbg_spread3(unsigned long long v)
{
    v = (v | v << 32) & 0x001f00000000ffffull;
    v = (v | v << 16) & 0x001f0000ff0000ffull;
    v = (v | v << 8) & 0x100f00f00f00f00full;
    v = (v | v << 4) & 0x10c30c30c30c30c3ull;
    return (v | v << 2) & 0x1249249249249249ull;
}

/* A root cube as a grid: centre, half size, low corner, cells per unit length,
 * and the margin (in 2^-30 of a cell) around a cell's faces that is not sure.
 *
 * The descent rounds each of its 21 centres, by at most 2^-53 A each, A the
 * largest coordinate's magnitude; the cell's arithmetic adds 2^-53 (A + 2 half)
 * and, relative, 2^-52, and 2^-31 of a cell.  A cell is half / 2^20 and a
 * coordinate below 2^21 cells, so that is below 25/8 A / half + 2 in 2^-30 of a
 * cell; the margin is 8 A / half + 16 or more. */
typedef struct {
    double cx, cy, cz, half, lx, ly, lz, inv;
    unsigned margin;
} NbgOctGrid;

NBG_OFN NbgOctGrid nbg_oct_grid(double cx, double cy, double cz, double half)
{
    NbgOctGrid g;
    g.cx = cx;
    g.cy = cy;
    g.cz = cz;
    g.half = half;
    g.lx = cx - half;
    g.ly = cy - half;
    g.lz = cz - half;
    g.inv = (double)(1 << (NBG_OCT_LEVELS - 1)) / half;
    const float a = (float)(fmax(fabs(cx), fmax(fabs(cy), fabs(cz))) / half) + 1.0f;
    /* otherwise, NaN included, nothing is sure */
    g.margin = a < 1e6f && half > 1e-250 && half < 1e250 ? (unsigned)(8.5f * a) + 17u : 1u << 30;
    return g;
}

NBG_OFN int nbg_oct_axis(double x, double lo, double inv, unsigned margin, unsigned long long *cell)
{
    const double v = (x - lo) * inv + 4194304.0; /* 2^22 + cells: the last bit is 2^-30 */
    unsigned long long b;
#if defined(__CUDA_ARCH__)
    b = (unsigned long long)__double_as_longlong(v);
#else
    memcpy(&b, &v, 8);
#endif
    const unsigned frac = (unsigned)b & 0x3fffffffu;
    *cell = (b >> 30) & 0x3fffffu;
    return (unsigned)(b >> 52) == 1023u + 22u && *cell < (1ull << NBG_OCT_LEVELS) && margin < (1u << 29) &&
           frac - margin < (1u << 30) - 2u * margin;
}

/* the path into key, or 0 when a coordinate's cell is not sure */
NBG_OFN int nbg_oct_cell(const NbgOctGrid &g, double x, double y, double z, unsigned long long &key)
{
    unsigned long long ix, iy, iz;
    const int sx = nbg_oct_axis(x, g.lx, g.inv, g.margin, &ix), sy = nbg_oct_axis(y, g.ly, g.inv, g.margin, &iy),
              sz = nbg_oct_axis(z, g.lz, g.inv, g.margin, &iz);
    key = nbg_spread3(ix) | nbg_spread3(iy) << 1 | nbg_spread3(iz) << 2;
    return sx && sy && sz;
}

#endif /* NBG_OCTANT_H */
