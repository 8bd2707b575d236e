"""Fixed-point positions (octree-cuda_gb300/csrc/fixed_axis.h, compiled with the
host compiler) against the binary64 formulas they stand for: output coordinates,
and cells of every level's nodes.  Wherever a position is called proven it must
agree; points on and one step beside every boundary are among those tried."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include <random>
#include "fixed_axis.h"
using namespace oc;

// cell of p at a node of `level` (grid cells of 128 per node), the reference's
// way: box minima by additions on the way down, then (p - min) / t
static long node_cell(double p, double mn, double side, unsigned depth, unsigned level, long path, long grid) {
    double m = mn, sz = side;
    long at = 0;
    for (unsigned l = depth; l > level; --l) {
        sz *= 0.5;
        at <<= 1;
        if (path >> (l - level - 1) & 1) { m = m + sz; at |= 1; }
    }
    const double t = ((m + sz) - m) / (double)grid;
    const double u = std::fmin((p - m) / t, (double)grid - 1.0);
    return u > -1.0 ? (long)u : -1;
}

int main(int argc, char** argv) {
    const double mn = std::atof(argv[1]), side = std::atof(argv[2]), scale = std::atof(argv[3]);
    const unsigned depth = (unsigned)std::atoi(argv[4]);
    const bool f32 = std::atoi(argv[5]) != 0;
    const double sf = 1.0 / scale;
    const FixedAxis a = make_fixed_axis(mn, side, sf, depth);
    const unsigned long fine_cells = 64ul << depth;
    std::mt19937_64 r(1);
    long bad = 0, tried = 0, known = 0, proven_cells = 0;
    auto point = [&](double p) {
        if (f32) {
            const float f = (float)p;
            p = (double)f;
            uint32_t b;
            std::memcpy(&b, &f, 4);
            // the value itself, or one with no place in the box
            if (std::fpclassify(f) == FP_NORMAL && widen_bits(b) != p) ++bad;
            if (!std::isfinite(f) && std::fabs(widen_bits(b)) < 3e38) ++bad;
        }
        uint64_t d;
        bool ok;
        ++tried;
        if (!fixed_difference(p, a.o, d)) {
            if (a.o.c == a.o.c && p > mn && p < mn + side * 0.999999) ++bad;   // points of the box have a position
            return;
        }
        const double want = std::floor((p - mn) * sf);
        const uint32_t v = fixed_units(d, a.out, ok);
        if (ok && (int32_t)v >= 0) {
            ++known;
            if ((double)v != want) ++bad;
        }
        const uint32_t c = fixed_units(d, a.cell, ok);
        if (!ok || c >= fine_cells) return;
        ++proven_cells;
        for (unsigned level = 1; level <= depth; ++level) {
            // node of the level that holds the cell: 128 << (level - 1) finest cells wide
            const long path = c >> (6 + level), in = c & ((128l << (level - 1)) - 1);
            for (long grid = 8; grid <= 128; grid *= 2)
                if (node_cell(p, mn, side, depth, level, path, grid) != in * grid >> (6 + level)) ++bad;
        }
        if (node_cell(p, mn, side, depth, depth, 0, (long)(fine_cells >> 6)) != (long)(c >> 6)) ++bad;   // counting
    };
    auto around = [&](double p) {
        point(p);
        for (double q = p, s = p, i = 0; i < 3; ++i) {
            q = f32 ? (double)std::nextafter((float)q, INFINITY) : std::nextafter(q, INFINITY);
            s = f32 ? (double)std::nextafter((float)s, -INFINITY) : std::nextafter(s, -INFINITY);
            point(q);
            point(s);
        }
        for (double e = 1e-14; e < 1e-5; e *= 10) { point(p + e * side); point(p - e * side); }
    };
    for (int i = 0; i < 4000; ++i) {
        const double u = (double)(r() >> 11) * 0x1p-53;
        point(mn + side * u);
        around(mn + side / (double)fine_cells * (double)(r() % (fine_cells + 1)));
        around(mn + std::floor(side * u * sf) * scale);
    }
    around(mn);
    around(mn + side);
    for (double p : {-1e300, 1e300, mn - side, mn + 4 * side, 0.0, -0.0, 1e-40, (double)INFINITY, -(double)INFINITY,
                     (double)NAN})
        point(p);
    std::printf("%ld %ld %ld %ld\n", bad, tried, known, proven_cells);
    return 0;
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    if not shutil.which("g++"):
        pytest.skip("no host compiler")
    d = tmp_path_factory.mktemp("fixed_axis")
    (d / "t.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-I", os.path.join(ROOT, "octree-cuda_gb300", "csrc"),
                    str(d / "t.cpp"), "-o", str(d / "t")], check=True)
    return str(d / "t")


@pytest.mark.parametrize("f32", [0, 1])
@pytest.mark.parametrize("mn,side,scale,depth", [
    (0.0, 1.0, 0.001, 1), (0.0, 1.0, 0.001, 10), (-50.5, 101.0, 0.001, 7), (1e6, 100.0, 0.01, 9),
    (-4.7e6, 5000.0, 0.01, 10), (-3.3, 8.0, 1e-8, 5), (1e-3, 1e-4, 1e-9, 6), (123456.789, 2.0, 0.001, 10),
    (0.0, 1000.0, 1e-9, 8), (1e12, 10.0, 0.1, 4), (0.0, 1e-20, 1e-24, 3), (0.0, 3e9, 1.0, 10)])
def test_positions(program, mn, side, scale, depth, f32):
    out = subprocess.run([program, repr(mn), repr(side), repr(scale), str(depth), str(f32)], check=True,
                         capture_output=True, text=True).stdout
    bad, tried, known, cells = map(int, out.split())
    assert tried > 100_000 and bad == 0
    if mn == 0.0 and side == 1.0 and not f32:   # an ordinary box: about all but the points put on boundaries
        assert known > tried * 0.5 and cells > tried * 0.5


# The same points through fixed_cell: the cell holds in every grid of cells wider than the boundary it names, also
# for points at both ends of the box and beyond its upper one, which the formulas clamp.
CELLS = r"""
        uint32_t low = 0;
        const uint32_t c = fixed_cell(d, a.cell, (uint32_t)fine_cells, low);
        if (c >= fine_cells) ++bad;
        if (a.cell.room == 0 && !low && p > mn + side / 4 && p < mn + side * 0.75) ++bad;   // nothing is proven
        if (!low) ++proven_cells;
        for (unsigned level = 1; level <= depth; ++level) {
            const long path = c >> (6 + level), in = c & ((128l << (level - 1)) - 1);
            for (long grid = 8; grid <= 128; grid *= 2)
                if (low < ((128l << (level - 1)) / grid) &&
                    node_cell(p, mn, side, depth, level, path, grid) != in * grid >> (6 + level)) ++bad;
        }
        if (low < 64 && node_cell(p, mn, side, depth, depth, 0, (long)(fine_cells >> 6)) != (long)(c >> 6)) ++bad;
    };
"""


@pytest.fixture(scope="module")
def cells_program(tmp_path_factory):
    if not shutil.which("g++"):
        pytest.skip("no host compiler")
    d = tmp_path_factory.mktemp("fixed_cells")
    begin = PROGRAM.index("        const uint32_t c = fixed_units(d, a.cell, ok);")
    end = PROGRAM.index("    auto around")
    (d / "t.cpp").write_text(PROGRAM[:begin] + CELLS + PROGRAM[end:])
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-I", os.path.join(ROOT, "octree-cuda_gb300", "csrc"),
                    str(d / "t.cpp"), "-o", str(d / "t")], check=True)
    return str(d / "t")


@pytest.mark.parametrize("f32", [0, 1])
@pytest.mark.parametrize("mn,side,depth", [
    (0.0, 1.0, 1), (0.0, 1.0, 10), (0.0, 4096.0, 9), (-50.5, 101.0, 7), (1e6, 100.0, 9), (-4.7e6, 5000.0, 10),
    (437000.0, 51.2, 6), (123456.78, 3000.32, 9), (5412345.67, 25.6, 5), (1e12, 10.0, 4), (0.0, 3e9, 10)])
def test_cells_beside_boundaries(cells_program, mn, side, depth, f32):
    out = subprocess.run([cells_program, repr(mn), repr(side), "0.01", str(depth), str(f32)], check=True,
                         capture_output=True, text=True).stdout
    bad, tried, _, cells = map(int, out.split())
    assert tried > 100_000 and bad == 0
