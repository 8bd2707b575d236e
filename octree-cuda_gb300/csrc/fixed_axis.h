// Positions on an axis in fixed point, on the host and the device.
//
// The reference takes cells and output coordinates from binary64 formulas,
// floor of (p - min) times or over something (mapPointToGrid,
// OctreeLibrary/src/kernel/kernel_helpers.cuh:10-25; point_distributing.cuh:
// 245-247).  Here one binary64 addition turns a coordinate into an integer, and
// everything after it is integer: with 2^k > side, t = p + (2^k - min) lies in
// [2^k, 2^(k+1)) for every point of the box, so that its 52 mantissa bits are
// (p - min) in steps of 2^(k-52).  (Points below or far above the box, infinite
// and NaN ones have another exponent.)  The upper 64 bits of the product with
// a 64-bit factor are the position in 32.32 fixed point.
//
// Its integer part is what the binary64 formula gives unless the fraction lies
// within `e` of an integer: e covers the rounding of t and of 2^k - min, the
// truncated parts of the product and what rounding moves the formula itself.
// The caller evaluates the formula where that is not so.
#pragma once

#include <cmath>
#include <cstdint>
#include <cstring>
#include <limits>

#if defined(__CUDACC__)
#define OC_FIXED_FN __host__ __device__ __forceinline__
#else
#define OC_FIXED_FN inline
#endif

namespace oc {

struct FixedOrigin {
    double c;       // 2^k - min; NaN where no position can be had this way
    uint32_t top;   // high word of 2^k
};

// Units of one kind (output steps, cells) per coordinate unit.
struct FixedScale {
    uint32_t lo, hi;    // units * 2^(k + 32)
    uint32_t e, room;   // proven: e <= fraction < 2^32 - e; room = 2^32 - 2 e (0: never)
};

inline FixedOrigin make_fixed_origin(double mn, double side) {
    FixedOrigin o{std::numeric_limits<double>::quiet_NaN(), 0};
    if (!(side > 1e-15 && side < 1e30) || !(std::fabs(mn) < 1e30)) return o;
    int k = 0;
    std::frexp(side, &k);   // side < 2^k
    o.c = std::ldexp(1.0, k) - mn;
    o.top = (uint32_t)(k + 1023) << 20;
    return o;
}

// formula: what rounding can move the binary64 formula, in units.
inline FixedScale make_fixed_scale(const FixedOrigin& o, double units, double formula) {
    FixedScale s{0, 0, 1u << 31, 0};
    if (!(o.c == o.c)) return s;
    const int k = (int)(o.top >> 20) - 1023;
    const double factor = std::ldexp(units, k + 32);
    if (!(factor >= 1.0 && factor < 18446744073709551616.0)) return s;
    // half a step of t, half an ulp of c, then truncations of under 8 * 2^-32 units
    const double err = units * (std::ldexp(1.0, k - 53) + std::ldexp(std::fabs(o.c), -53)) + formula;
    const double e = std::ceil(err * 4294967296.0 * 1.001) + 8.0;
    if (!(e < 2147483648.0)) return s;
    const uint64_t f = (uint64_t)factor;
    s.lo = (uint32_t)f;
    s.hi = (uint32_t)(f >> 32);
    s.e = (uint32_t)e;
    s.room = 0u - 2u * s.e;
    return s;
}

// A binary32 value (its bits) as binary64 without a conversion instruction:
// zero and denormals come out below 2^-126, infinity and NaN as 2^128 and
// more, which is outside every box that has an origin.
OC_FIXED_FN double widen_bits(uint32_t b) {
    const uint64_t v = (uint64_t)(((b & 0x7FFFFFFFu) >> 3) + (896u << 20) | (b & 0x80000000u)) << 32 | (uint32_t)(b << 29);
    double d;
    memcpy(&d, &v, 8);
    return d;
}

// p - min in steps of 2^(k-64); false where p has no position.
OC_FIXED_FN bool fixed_difference(double p, const FixedOrigin& o, uint64_t& d) {
#if defined(__CUDA_ARCH__)
    const double t = __dadd_rn(p, o.c);
#else
    const double t = p + o.c;
#endif
    uint64_t v;
    memcpy(&v, &t, 8);
    const uint32_t hi = (uint32_t)(v >> 32) - o.top;
    d = ((uint64_t)hi << 32 | (uint32_t)v) << 12;
    return hi < (1u << 20);
}

// Position in units; proven says that the binary64 formula gives the same.
OC_FIXED_FN uint32_t fixed_units(uint64_t d, const FixedScale& s, bool& proven) {
    const uint32_t dl = (uint32_t)d, dh = (uint32_t)(d >> 32);
    const uint64_t u = (uint64_t)dh * s.hi + (uint32_t)((uint64_t)dh * s.lo >> 32) + (uint32_t)((uint64_t)dl * s.hi >> 32);
    proven = (uint32_t)u - s.e < s.room;
    return (uint32_t)(u >> 32);
}

// Finest cell of a position, of `cells` on the axis.  low becomes the lowest set
// bit of a boundary between cells, if greater, that the position lies so near to
// that the binary64 formulas could put it on either side (2^31 where nothing is
// proven on the axis).  The cell of a coarser grid, 2^j finest cells wide, is the
// upper bits unless the boundary is a multiple of 2^j.  Below the first boundary
// and above the last the formulas clamp to the outermost cells of every grid.
OC_FIXED_FN uint32_t fixed_cell(uint64_t d, const FixedScale& s, uint32_t cells, uint32_t& low) {
    const uint32_t dl = (uint32_t)d, dh = (uint32_t)(d >> 32);
    const uint64_t u = (uint64_t)dh * s.hi + (uint32_t)((uint64_t)dh * s.lo >> 32) + (uint32_t)((uint64_t)dl * s.hi >> 32);
    const uint32_t f = (uint32_t)u;
    uint32_t c = (uint32_t)(u >> 32);
    if (f - s.e >= s.room || c >= cells) {
        const uint32_t b = s.room == 0 ? 1u << 31 : c + (f >> 31) < cells ? c + (f >> 31) : 0u;
        if ((b & (0u - b)) > low) low = b & (0u - b);
        if (c >= cells) c = cells - 1;
    }
    return c;
}

// One axis of the cloud's cube: output coordinates and the finest subsampling
// cells (those of 128^3 grids in the nodes of level 1, 64 per counting cell).
struct FixedAxis {
    FixedOrigin o;
    FixedScale out, cell;
};

struct FixedGrid {
    FixedAxis ax[3];
    uint32_t cells;   // finest cells per axis
};

// sf: output steps per unit; depth: of the tree.  The output formula rounds
// its difference and its product, 2^-52 of the position together.  A node's box minimum comes from
// at most `depth` additions of binary64, its cell size from two more roundings
// of numbers up to M = max(|mn|, |mn + side|, side), and the cell formula adds
// the rounding of p - min and of the quotient: together under
// (depth + 8) * 2^-52 * M in coordinate units; twice that is allowed for.
inline FixedAxis make_fixed_axis(double mn, double side, double sf, uint32_t depth) {
    FixedAxis a;
    a.o = make_fixed_origin(mn, side);
    const double cells = (double)(64ull << depth), per_unit = cells / side;
    const double M = std::fmax(std::fmax(std::fabs(mn), std::fabs(mn + side)), side);
    a.out = make_fixed_scale(a.o, sf, std::ldexp(sf * side, -50));
    a.cell = make_fixed_scale(a.o, per_unit, std::ldexp((depth + 8.0) * M * per_unit + cells, -51));
    return a;
}

}   // namespace oc
