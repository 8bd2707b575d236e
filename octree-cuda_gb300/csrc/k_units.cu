// Subsampling by octants (power-of-two subsampling grids from 8 to 128).
//
// A child lies in one octant of its parent, so the cells of a node's S^3 grid
// that its candidates fall in are the cells of that octant: nodes split into
// independent units (node, child octant) of at most (S/2)^3 cells, and a level
// is a flat list of units that blocks take in order.  Per unit:
//
//   pass A  every candidate's cell is read from its cell word (below) and
//           marked in a dense bitmap of the octant in shared memory
//   ranks   a prefix sum of the bitmap gives every occupied cell its rank
//   place   the unit's cells follow those of the node's earlier units: it
//           waits for their counts (earlier units were taken earlier, so the
//           oldest unit never waits and the wait always ends)
//   pass B  per candidate: selection key minimum and packed colour sum of its
//           cell, in L2 by reductions that return nothing
//   emit    colours per cell
//
// Cell words.  A candidate's cell in a node is the cell its position in the
// cloud's cube gives at that node's resolution, unless rounding of the
// reference's binary64 formula could decide otherwise: distribution tells the
// points for which it could, and at which levels (fixed_cell, kWordEdge), and
// stores the point's cell in its leaf's parent; each level's output stores its
// own cell, and the parent's is that, halved.  Where the formula decides, the
// cell is evaluated from the cloud point in binary64, once: the word keeps it
// for the unit's later passes.  When that
// lands outside the unit (a point on an octant boundary that the two levels
// round differently; common where coordinates are multiples of a scale and the
// box is too) kErrForeign is set, and the levels from this one on are done again
// with such points handed to the units of their cells (k_foreign).
//
// What a level writes per output point: cloud index, cell word and (averaged
// modes) colour, 8 to 16 bytes instead of the 18-byte record; k_place_units
// makes the records of all levels at the end from the cloud points.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <map>
#include <mutex>
#include <utility>

#include "device_common.cuh"
#include "kernels.h"

#ifndef OC_UNITS_PART
#define OC_UNITS_PART 0
#endif

namespace oc {

namespace {

// Blocks of a level (T threads): two of 640 per SM hide each other's barriers;
// one of 1024 has the whole shared memory for its unit's cells; two of 768 for
// distance weighting, whose emit runs on instructions and loads alone.
constexpr int unit_blocks(int T) { return T == 1024 ? 1 : 2; }
constexpr uint32_t kFieldBits = 7;   // coordinates of a cell word: x | y << 7 | z << 14

__device__ __forceinline__ uint32_t fields(uint32_t x, uint32_t y, uint32_t z) {
    return x | (y << kFieldBits) | (z << (2 * kFieldBits));
}

__device__ __forceinline__ uint64_t load_acquire(const uint64_t* p) {
    uint64_t v;
    asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}

__device__ __forceinline__ void store_release(uint64_t* p, uint64_t v) {
    asm volatile("st.release.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

// Waits until *p is not 0; gives up after `limit` clock cycles (a negative
// limit: at once) and returns 0.
__device__ __forceinline__ uint64_t wait_nonzero(const uint64_t* p, long long limit) {
    uint64_t v = limit < 0 ? 0 : load_acquire(p);
    if (v || limit < 0) return v;
    const long long t0 = clock64();
    while (!(v = load_acquire(p)))
        if (clock64() - t0 > limit) return 0;
    return v;
}

// Cell of a cloud point in the node's grid by the binary64 formula
// (mapPointToGrid, kernel_helpers.cuh:10-25), as coordinates.
__device__ __noinline__ uint32_t exact_cell(const UnitLevelArgs& a, const SubNode& nd, uint32_t idx) {
    Coord co[3];
    uint32_t col[3];
    const uint8_t* p = a.cloud + (uint64_t)idx * a.stride;
    const uint32_t G = 1u << a.s;
    int c[3];
    float u;
    if (a.float_input) {
        load_point<true>(p, co, col);
        for (int k = 0; k < 3; ++k) c[k] = axis_cell<true>(co[k], nd.ax[k], G, u);
    } else {
        load_point<false>(p, co, col);
        for (int k = 0; k < 3; ++k) c[k] = axis_cell<false>(co[k], nd.ax[k], G, u);
    }
    if ((c[0] | c[1] | c[2]) < 0) {
        atomicOr(a.err, kErrBelowBox);
        for (int k = 0; k < 3; ++k) c[k] = max(c[k], 0);
    }
    return fields((uint32_t)c[0], (uint32_t)c[1], (uint32_t)c[2]);
}

__device__ __forceinline__ uint64_t pack_colour(uint16_t r, uint16_t g, uint16_t b) {
    return (uint64_t)r | ((uint64_t)g << 16) | ((uint64_t)b << 32);
}

// The unit in work: where its candidates are and how their words map to cells
// of its box (side 2^b at (x0, y0, z0) of the node's grid).
struct Unit {
    uint32_t node, octant, part, index;
    uint32_t staged, first, last, q0;
    uint32_t large, map;   // a large leaf (k_large_mark); word offset of its bitmap and ranks
    uint32_t cnt;
    uint32_t b;
    uint32_t base;    // fields(x0, y0, z0)
    uint32_t open;    // faces of the box inside the node: bits x low, x high, y, z
    uint64_t start;
};

__device__ __forceinline__ Unit load_unit(const UnitLevelArgs& a, uint32_t u) {
    const UnitEntry e = a.units[u];
    Unit v;
    v.node = e.node;
    v.octant = e.flags & 7;
    v.part = (e.flags >> 3) & 15;
    v.staged = (e.flags >> 7) & 1;
    v.first = (e.flags >> 8) & 1;
    v.last = (e.flags >> 9) & 1;
    v.index = (e.flags >> 10) & 63;
    v.q0 = (e.flags >> 16) & 15;
    v.large = (e.flags >> 20) & 1;
    v.map = e.map;
    v.start = e.src;
    v.cnt = e.count;
    if (v.staged) {
        const uint32_t ii = e.src;
        v.cnt = a.out_points[ii];
        v.start = a.stage_off[ii];
        if (v.part) {   // the child's own octant, contiguous in its output
            const uint32_t o2 = v.part - 8;
            const uint32_t lo = a.oct_off[(uint64_t)ii * 8 + o2];
            const uint32_t hi = o2 == 7 ? v.cnt : a.oct_off[(uint64_t)ii * 8 + o2 + 1];
            v.start += lo;
            v.cnt = hi - lo;
        }
    }
    const uint32_t h = a.s - 1;
    uint32_t x = ((v.octant >> 2) & 1) << h, y = ((v.octant >> 1) & 1) << h, z = (v.octant & 1) << h;
    v.b = h;
    if (v.part) {
        const uint32_t o2 = v.part - 8;
        v.b = h - 1;
        x |= ((o2 >> 2) & 1) << v.b;
        y |= ((o2 >> 1) & 1) << v.b;
        z |= (o2 & 1) << v.b;
    }
    v.base = fields(x, y, z);
    const uint32_t side = 1u << v.b, S = 1u << a.s;
    v.open = (x > 0 ? 1u : 0u) | (x + side < S ? 2u : 0u) | (y > 0 ? 4u : 0u) | (y + side < S ? 8u : 0u) |
             (z > 0 ? 16u : 0u) | (z + side < S ? 32u : 0u);
    return v;
}

// Brings the whole 16-byte words of [p, p + bytes) into L2.
__device__ __forceinline__ void prefetch_l2(const void* p, uint64_t bytes) {
    const uint64_t g = __cvta_generic_to_global(p), first = (g + 15) & ~15ull, end = (g + bytes) & ~15ull;
    if (first < end)
        asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(first), "r"((uint32_t)(end - first)) : "memory");
}

// The candidates of a unit that some block will take soon: passes A and B wait
// for their loads (a third of the time of the warps).
// 12.3M points 1.620 -> 1.600 ms, 25.8M intra-cell 3.03 -> 2.99, 119.7M the
// same; distance weighting reads points all over the cloud and loses 1% by it.
template <int kColor>
__device__ __forceinline__ void prefetch_unit(const UnitLevelArgs& a, uint32_t u) {
    const Unit v = load_unit(a, u);
    if (v.large) return;
    prefetch_l2((v.staged ? a.stage_word : a.leaf_word) + v.start, (uint64_t)v.cnt * 4);
    prefetch_l2((v.staged ? a.stage_lut : a.leaf_lut) + v.start, (uint64_t)v.cnt * 4);
    if (kColor) {
        if (v.staged) prefetch_l2(a.stage_col + v.start, (uint64_t)v.cnt * 8);
        else prefetch_l2(a.leaf_rec + v.start * 18, (uint64_t)v.cnt * 18);
    }
}

// Bits of the box's faces a cell lies on (as Unit::open).
__device__ __forceinline__ uint32_t faces_of(uint32_t x, uint32_t y, uint32_t z, uint32_t m0) {
    return (x == 0 ? 1u : 0u) | (x == m0 ? 2u : 0u) | (y == 0 ? 4u : 0u) | (y == m0 ? 8u : 0u) | (z == 0 ? 16u : 0u) |
           (z == m0 ? 32u : 0u);
}

// Appends the cells of the lanes with `face` to the node's face list (every
// lane of the warp calls it): rank, word, and packed colour sum or partial.
__device__ __forceinline__ void append_faces(const UnitLevelArgs& a, uint32_t node, uint64_t off, uint32_t rank,
                                             uint32_t word, uint64_t sum, bool face) {
    const uint32_t lane = threadIdx.x & 31, m = __ballot_sync(0xffffffffu, face);
    if (!m) return;
    uint32_t first = 0;
    if (lane == 0) first = atomicAdd(&a.node_state[node].faces, (uint32_t)__popc(m));
    first = __shfl_sync(0xffffffffu, first, 0);
    if (face) {
        const uint64_t f = off + first + __popc(m & ((1u << lane) - 1u));
        a.faces[f] = make_uint2(rank, word);
        a.face_sum[f] = sum;
    }
}

// Words of a unit's bitmap, and in the map of a large leaf (bitmap, one word
// more, ranks) the place of what its blocks share: candidates, whether one lies
// beside a boundary, and the unit's first candidate in the node.
__host__ __device__ constexpr uint32_t bitmap_words(uint32_t b) { return 3 * b > 5 ? 1u << (3 * b - 5) : 1u; }
__host__ __device__ constexpr uint32_t large_state(uint32_t b) { return 2 * bitmap_words(b) + 4; }

struct BlockShared {
    Unit un;
    uint32_t warp[32];
    uint32_t unit, unsafe, foreign, rank0, cand0, included, next, fail, redo, stop;
    int32_t delta;
    uint64_t off, level_base;
};

// Bytes a cell takes in shared memory: selection key, colour sum (weighted:
// candidates), word.
__host__ __device__ constexpr uint32_t cell_bytes(int color, bool random) {
    return (random ? 8u : 4u) + (color == 3 ? 4u : color >= 1 ? 8u : 0u) + 4u;
}

// Distance weighting: the point ranges a group of lanes walks for its cell, as {end in the cell's list, first point - begin in the list}.
constexpr uint32_t kWeightLanes = 4;   // per cell
constexpr int kWeightThreads = 768;
struct WeightShared {
    uint2 rows[kWeightThreads / kWeightLanes][9];
};

// Units of many candidates per cell have shared sums of 32 bits per colour: the
// packed ones (exact up to 257 candidates) would mostly have to be done again in
// global memory, where the cells' reductions queue up (grids of 8: 3M
// binary64 points 1.23 ms, before octants 0.87).  32 bits hold 16.8M candidates of 8-bit colours.
__device__ __forceinline__ bool dense_unit(uint32_t candidates, uint32_t cells) {
    return candidates / 24 > cells && candidates < (1u << 23);
}

// Node-grid cell of a candidate without the proof, as coordinates; foreign
// when it is not the unit's.
__device__ __forceinline__ uint32_t node_cell(const UnitLevelArgs& a, const Unit& un, uint32_t idx, bool& foreign) {
    const uint32_t f = exact_cell(a, a.nodes[un.node], idx);
    const uint32_t x = f & 127, y = (f >> kFieldBits) & 127, z = f >> (2 * kFieldBits), b = un.b;
    const uint32_t h = a.s - 1;
    const bool other = (((x >> h) << 2) | ((y >> h) << 1) | (z >> h)) != un.octant;
    const bool part = un.part && ((((x >> b) & 1) << 2) | (((y >> b) & 1) << 1) | ((z >> b) & 1)) != un.part - 8;
    foreign = other || part;
    return f;
}

// Whether a word's cell may differ from the formula's in the level's grids, or
// was evaluated for another grid (a leaf's, of a resident tree).
__device__ __forceinline__ bool unproven(const UnitLevelArgs& a, uint32_t w) {
    return ((w >> kWordEdge) & 31u) > a.level + 6 - a.s || ((w & kWordResolved) && ((w >> kWordGrid) & 7u) != a.s);
}

// Cell of an unproven candidate, evaluated once per node; the unit that reads
// the candidate leaves it in the word.
__device__ __forceinline__ uint32_t resolved_word(const UnitLevelArgs& a, const Unit& un, uint32_t* word, uint32_t w,
                                                  uint32_t idx) {
    if ((w & kWordResolved) && ((w >> kWordGrid) & 7u) == a.s) return w;
    bool foreign;
    const uint32_t f = node_cell(a, un, idx, foreign);
    w = f | (w & kWordEdges) | (a.s << kWordGrid) | kWordResolved | (foreign ? kWordForeign : 0u);
    *word = w;
    return w;
}

// The cell of candidate k, ~0 for a foreign one: k_foreign has handed it to the unit its
// cell is in, or the pass is repeated with that, from this level.
__device__ __noinline__ uint32_t unproven_cell(const UnitLevelArgs& a, const Unit& un, uint32_t k, uint32_t w) {
    const uint64_t at = un.start + k;
    w = resolved_word(a, un, (un.staged ? a.stage_word : a.leaf_word) + at, w, (un.staged ? a.stage_lut : a.leaf_lut)[at]);
    if (!(w & kWordForeign)) return w & kWordCell;
    if (!a.foreign_head) {
        a.err[1] = a.level;
        atomicOr(a.err, kErrForeign);
    }
    return ~0u;
}

// Calls get(cell as Box::cell takes it with its kWordEdge bits, cloud index, r |
// g << 16, b) for the points of other units whose cell lies in this one: the block's
// threads take the points of one segment after the other.
template <class Get>
__device__ __forceinline__ void foreign_points(const UnitLevelArgs& a, const Unit& un, uint32_t head, Get&& get) {
    for (uint32_t seg = head; seg;) {
        const uint4 h = a.foreign[seg - 1];
        for (uint32_t k = threadIdx.x; k < h.y; k += blockDim.x) {
            const uint4 e = a.foreign[seg + k];
            const uint32_t b = un.b, x = e.x & 127, y = (e.x >> kFieldBits) & 127, z = (e.x >> (2 * kFieldBits)) & 127;
            if (un.part && ((((x >> b) & 1) << 2) | (((y >> b) & 1) << 1) | ((z >> b) & 1)) != un.part - 8) continue;
            get(e.x, e.y, e.z, e.w);
        }
        seg = h.x;
    }
}

// Waits for the counts of the node's earlier units and the node's place
// (warp 0): where the unit's cells go; writes the node's totals with its last
// unit.
__device__ __forceinline__ void unit_place(const UnitLevelArgs& a, BlockShared& sh, uint32_t ui, uint32_t cells) {
    const Unit& un = sh.un;
    const uint32_t lane = threadIdx.x & 31;
    uint32_t r0 = 0, c0 = 0;
    bool ok = true;
    for (uint32_t q = lane; q < un.index; q += 32) {
        const uint64_t v = wait_nonzero(&a.unit_state[ui - 1 - q], a.wait_limit);
        ok = ok && v != 0;
        r0 += (uint32_t)v - 1;
        c0 += (uint32_t)(v >> 32);
    }
    uint64_t off1 = 0;
    if (lane == 0) off1 = wait_nonzero(&a.node_state[un.node].off1, a.wait_limit);
    ok = ok && (lane != 0 || off1 != 0);
    r0 = __reduce_add_sync(0xffffffffu, r0);
    c0 = __reduce_add_sync(0xffffffffu, c0);
    ok = __all_sync(0xffffffffu, ok);
    if (lane == 0) {
        if (!ok) atomicOr(a.err, kErrTimeout);
        const bool fail = !ok || off1 == ~0ull;
        const uint32_t ii = a.first_internal + un.node;
        uint32_t* oct = a.oct_off + (uint64_t)ii * 8;
        if (un.part == 0 || un.part == 8)
            for (uint32_t q = un.q0; q <= un.octant; ++q) oct[q] = fail ? 0u : r0;
        if (un.last) {
            const uint32_t total = fail ? 0u : r0 + cells;
            for (uint32_t q = un.octant + 1; q < 8; ++q) oct[q] = total;
            a.out_points[ii] = total;
            a.stage_off[ii] = fail ? 0u : sh.level_base + off1 - 1;
            a.node_state[un.node].points = c0 + sh.included;
        }
        a.unit_rank[ui] = r0;
        sh.rank0 = r0;
        sh.cand0 = c0;
        sh.off = off1 - 1;
        sh.fail = fail;
    }
}

// The dense bitmap of a unit's box (cell x | y << b | z << 2b) and the
// number of occupied cells before each of its words.  kB: b at compile time
// (0: any); Pre: the type of those numbers (32 bits for a unit of more than
// 65535 candidates).
template <int kB, class Pre>
struct Box {
    const uint32_t* bm;
    const Pre* pre;
    uint32_t bits;
    __device__ __forceinline__ uint32_t b() const { return kB ? (uint32_t)kB : bits; }
    __device__ __forceinline__ uint32_t m0() const { return (1u << b()) - 1u; }
    __device__ __forceinline__ uint32_t cell(uint32_t f) const {   // of coordinates with other bits around them
        const uint32_t s1 = kFieldBits - b();
        return (f & m0()) | ((f >> s1) & (m0() << b())) | ((f >> (2 * s1)) & (m0() << (2 * b())));
    }
    __device__ __forceinline__ uint32_t coordinates(uint32_t i) const {
        return fields(i & m0(), (i >> b()) & m0(), i >> (2 * b()));
    }
    __device__ __forceinline__ uint32_t rank(uint32_t i) const {
        return pre[i >> 5] + __popc(bm[i >> 5] & ((1u << (i & 31)) - 1u));
    }
    // Sum of get(rank) over the box's cells around (x, y, z): nine rows of up
    // to three cells, whose ranks follow each other.
    template <class Get>
    __device__ __forceinline__ uint64_t sum27(uint32_t x, uint32_t y, uint32_t z, Get&& get) const {
        const uint32_t xa = x ? x - 1 : 0u;
        const uint32_t nm = (2u << (min(x + 1, m0()) - xa)) - 1u;
        uint64_t e = 0;
#pragma unroll
        for (int dz = -1; dz <= 1; ++dz) {
#pragma unroll
            for (int dy = -1; dy <= 1; ++dy) {
                const uint32_t yy = y + dy, zz = z + dz;
                if (yy <= m0() && zz <= m0()) {
                    const uint32_t i = xa | (yy << b()) | (zz << (2 * b())), w = i >> 5;
                    const uint32_t lo = bm[w], sh = i & 31u;
                    // (a row of 32 cells or fewer lies in one word)
                    const uint32_t t = (kB == 5 ? lo >> sh : __funnelshift_r(lo, bm[w + 1], sh)) & nm;
                    const uint32_t r = pre[w] + __popc(lo & ((1u << sh) - 1u));
                    if (t) e += get(r);
                    if (t & (t - 1)) e += get(r + 1);
                    if (t == 7) e += get(r + 2);
                }
            }
        }
        return e;
    }
};

// floor(sum / weight) of weighted colours of 8 bits: a float quotient is off
// by less than 2^-14, so that its integer part is off by at most one.
__device__ __forceinline__ uint32_t weighted_mean(uint64_t sum, uint64_t weight) {
    uint32_t q = (uint32_t)__fdividef(__ull2float_rn(sum), __ull2float_rn(weight));
    const int64_t rem = (int64_t)(sum - (uint64_t)q * weight);
    if (rem < 0) --q;
    else if ((uint64_t)rem >= weight) ++q;
    return q;
}

// Position of a cloud point in the node's grid, in cell units: the weight
// measures the distance from the point itself to each neighbour cell centre
// (kernel_inter_cell_filtering.cuh:171-176).
__device__ __forceinline__ float4 cell_units(const UnitLevelArgs& a, const SubNode& nd, uint32_t idx) {
    Coord co[3];
    uint32_t col[3];
    float4 v;
    const uint8_t* p = a.cloud + (uint64_t)idx * a.stride;
    if (a.float_input) {
        gather_point<true, false>(p, co, col);
        v.x = point_units<true>(co[0], nd.ax[0]);
        v.y = point_units<true>(co[1], nd.ax[1]);
        v.z = point_units<true>(co[2], nd.ax[2]);
    } else {
        gather_point<false, false>(p, co, col);
        v.x = point_units<false>(co[0], nd.ax[0]);
        v.y = point_units<false>(co[1], nd.ax[1]);
        v.z = point_units<false>(co[2], nd.ax[2]);
    }
    return v;
}

// The emit of a distance-weighted unit, whose candidates are grouped by cell:
// four lanes per cell.  The points of a row of up to three cells follow each
// other, so a cell's points are at most nine ranges: the lanes look them up,
// the ranges become one list by a prefix sum, and the lanes walk it four
// points at a time, which spreads a cell's points evenly whatever their cells
// hold.  (A lane per cell, or lanes sharing each neighbour's points, waits
// for the longest list: the weight of a pair costs about 45 instructions.)
// Colours are of 8 bits here: the cloud's, or means of those.
// cur: past each cell's last candidate of the unit; sh.next counts from the
// first cell to do up to `cells`.
template <bool kLocal, int kB, class Pre>
__device__ __forceinline__ void weighted_emit(const UnitLevelArgs& a, BlockShared& sh, const Box<kB, Pre>& box,
                                              const uint32_t* l_word, const uint32_t* cur, uint32_t cells, uint64_t oo,
                                              WeightShared& ws) {
    const uint32_t tid = threadIdx.x, lane = tid & 31;
    const Unit& un = sh.un;
    const uint64_t c0 = sh.off + sh.cand0;   // the unit's first candidate in the level's scratch
    auto cell_end = [&](uint32_t r) { return kLocal ? cur[r] : __ldcg(cur + r); };
    constexpr uint32_t kG = kWeightLanes;
    const uint32_t m0 = box.m0(), b = box.b(), g = lane / kG, s = lane % kG;
    uint2* rows = ws.rows[tid / kG];
    const uint32_t x0 = un.base & 127, y0 = (un.base >> kFieldBits) & 127, z0 = un.base >> (2 * kFieldBits);
    for (;;) {
        uint32_t first = 0;
        if (lane == 0) first = atomicAdd(&sh.next, 32u / kG);
        first = __shfl_sync(0xffffffffu, first, 0);
        if (first >= cells) break;
        const uint32_t r = first + g;
        const bool act = r < cells;
        uint32_t w = 0, x = 0, y = 0, z = 0;
        if (act) {
            w = kLocal ? l_word[r] : a.stage_word[oo + r];
            x = w & m0;
            y = (w >> kFieldBits) & m0;
            z = (w >> (2 * kFieldBits)) & m0;
        }
        const uint32_t xa = x ? x - 1 : 0u;
        const uint32_t nm = (2u << (min(x + 1, m0) - xa)) - 1u;
        // the lanes' rows s, s + kG, ... of the nine, one list after the other
        constexpr uint32_t kR = (9 + kG - 1) / kG;
        uint32_t from[kR], len[kR], sum = 0;
#pragma unroll
        for (uint32_t q = 0; q < kR; ++q) {
            const uint32_t k = s + q * kG, yy = y + k % 3 - 1, zz = z + k / 3 - 1;
            from[q] = len[q] = 0;
            if (act && k < 9 && yy <= m0 && zz <= m0) {
                const uint32_t i = xa | (yy << b) | (zz << (2 * b));
                const uint32_t t = __funnelshift_r(box.bm[i >> 5], box.bm[(i >> 5) + 1], i) & nm;
                if (t) {
                    const uint32_t n = box.rank(i);
                    from[q] = n ? cell_end(n - 1) : 0u;
                    len[q] = cell_end(n + __popc(t) - 1) - from[q];
                }
            }
            sum += len[q];
        }
        uint32_t incl = sum;
#pragma unroll
        for (uint32_t o = 1; o < kG; o <<= 1) {
            const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o, kG);
            if (s >= o) incl += v;
        }
        const uint32_t total = __shfl_sync(0xffffffffu, incl, kG - 1, kG);
        uint32_t run = incl - sum;
#pragma unroll
        for (uint32_t q = 0; q < kR; ++q) {
            // (entries in lane order: those of lane s follow lane s - 1's; lane 0 has one more when 9 % kG is 1)
            const uint32_t slot = s * (9 / kG) + min(s, 9 % kG) + q;
            if (s + q * kG < 9) rows[slot] = make_uint2(run + len[q], from[q] - run);
            run += len[q];
        }
        __syncwarp();
        uint64_t sr = 0, sg = 0, sb = 0, sw = 0;
        const float cx = __fadd_rn((float)(x0 + x), 0.5f), cy = __fadd_rn((float)(y0 + y), 0.5f),
                    cz = __fadd_rn((float)(z0 + z), 0.5f);
        uint2 e = rows[0];
        const float4* pts = a.csr_pts + c0;
        for (uint32_t p = s, k = 0; p < total; p += kG) {
            while (p >= e.x) e = rows[++k];
            const float4 v = pts[e.y + p];
            const uint32_t c = __float_as_uint(v.w);
            const uint32_t wq = weight_at(v.x, v.y, v.z, cx, cy, cz);
            sr += (uint64_t)wq * (c & 0xFFu);
            sg += (uint64_t)wq * ((c >> 8) & 0xFFu);
            sb += (uint64_t)wq * (c >> 16);
            sw += wq;
        }
#pragma unroll
        for (uint32_t o = kG / 2; o >= 1; o >>= 1) {
            sr += __shfl_xor_sync(0xffffffffu, sr, o);
            sg += __shfl_xor_sync(0xffffffffu, sg, o);
            sb += __shfl_xor_sync(0xffffffffu, sb, o);
            sw += __shfl_xor_sync(0xffffffffu, sw, o);
        }
        const bool face = act && (faces_of(x, y, z, m0) & un.open) != 0;
        // three lanes divide (the weight of the cell's own points is never 0)
        uint32_t c = 0;
        if (act && !face && s < 3) c = weighted_mean(s == 0 ? sr : s == 1 ? sg : sb, sw);
        const uint32_t c1 = __shfl_sync(0xffffffffu, c, 1, kG), c2 = __shfl_sync(0xffffffffu, c, 2, kG);
        uint64_t slot = 0;
        if (face && s == 0) {
            slot = atomicAdd(reinterpret_cast<unsigned long long*>(a.partials), 1ull);
            if (slot < a.partial_cap) {
                a.partial[slot * 4 + 0] = sr;
                a.partial[slot * 4 + 1] = sg;
                a.partial[slot * 4 + 2] = sb;
                a.partial[slot * 4 + 3] = sw;
            } else {
                a.err[1] = a.level;   // more face cells than there is room for: the level again, with more
                atomicOr(a.err, kErrPartials);
                slot = 0;
            }
        }
        if (act && !face && s == 0) a.stage_col[oo + r] = pack_colour((uint16_t)c, (uint16_t)c1, (uint16_t)c2);
        append_faces(a, un.node, sh.off, sh.rank0 + r, w, slot, face && s == 0);
        __syncwarp();   // the rows are written for the next cells
    }
}

// A distance-weighted unit after pass B: its candidates grouped by cell, and the emit.
template <int T, bool kRandom, int kB, bool kLocal, bool kOther, class Pre>
__device__ __forceinline__ void unit_weighted(const UnitLevelArgs& a, BlockShared& sh, const Box<kB, Pre>& box,
                                              const uint64_t* l_key, const uint32_t* l_word, uint32_t* l_cnt,
                                              uint32_t cells, const int (&keep)[4], uint64_t so, uint64_t oo,
                                              WeightShared& ws) {
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const Unit& un = sh.un;
    const uint32_t* l_idx = reinterpret_cast<const uint32_t*>(l_key);
    // ---- exclusive scan of the cells' counts, in place: the cursor of each
    // cell (first its first candidate, in the end one past its last)
    uint32_t* cur = kLocal ? l_cnt : a.csr_count + so;
    {
        const uint32_t per = (cells + T - 1) / T, r0 = min(tid * per, cells), r1 = min(r0 + per, cells);
        uint32_t sum = 0;
        for (uint32_t r = r0; r < r1; ++r) sum += kLocal ? cur[r] : __ldcg(cur + r);
        uint32_t incl = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= (uint32_t)o) incl += y;
        }
        if (lane == 31) sh.warp[warp] = incl;
        __syncthreads();
        uint32_t run = incl - sum;
        for (uint32_t q = 0; q < warp; ++q) run += sh.warp[q];
        for (uint32_t r = r0; r < r1; ++r) {
            const uint32_t n = kLocal ? cur[r] : __ldcg(cur + r);
            if (kLocal) cur[r] = run;
            else __stcg(cur + r, run);
            run += n;
        }
        __syncthreads();
    }
    const uint64_t c0 = sh.off + sh.cand0;   // the unit's first candidate in the level's scratch
    {
        const SubNode& nd = a.nodes[un.node];
        const uint32_t cnt = un.cnt;
        const bool staged = un.staged;
        const uint32_t shift = staged ? 1u : kFieldBits - a.s;
        const uint64_t start = un.start;
        const uint32_t* src_word = (staged ? a.stage_word : a.leaf_word) + start;
        const uint32_t* src_lut = (staged ? a.stage_lut : a.leaf_lut) + start;
        for (uint32_t k0 = tid, it = 0; k0 < cnt; k0 += 4 * T, it += 4) {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const uint32_t k = k0 + j * T;
                if (k >= cnt) break;
                const uint32_t idx = src_lut[k];
                int i = keep[j];
                if (it) {
                    i = -1;
                    const uint32_t w = src_word[k];
                    uint32_t f = w >> shift;
                    bool mine = true;
                    if ((w & kWordEdges) && unproven(a, w)) {
                        f = unproven_cell(a, un, k, w);
                        mine = f != ~0u;
                    }
                    if (mine) i = (int)box.cell(f);
                }
                if (i < 0) continue;
                float4 v = cell_units(a, nd, idx);
                uint32_t c;
                if (staged) {
                    const uint2 q = *reinterpret_cast<const uint2*>(a.stage_col + start + k);
                    c = (q.x & 0xFFu) | ((q.x >> 8) & 0xFF00u) | (q.y << 16);
                } else {
                    const uint16_t* q = reinterpret_cast<const uint16_t*>(a.leaf_rec + (start + k) * 18 + 12);
                    c = (uint32_t)q[0] | ((uint32_t)q[1] << 8) | ((uint32_t)q[2] << 16);
                }
                v.w = __uint_as_float(c);
                a.csr_pts[c0 + atomicAdd(cur + box.rank((uint32_t)i), 1u)] = v;
            }
        }
        if (kOther && sh.foreign)
            foreign_points(a, un, sh.foreign, [&](uint32_t f, uint32_t idx, uint32_t rg, uint32_t bl) {
                float4 v = cell_units(a, nd, idx);
                v.w = __uint_as_float((rg & 0xFFu) | ((rg >> 8) & 0xFF00u) | (bl << 16));
                a.csr_pts[c0 + atomicAdd(cur + box.rank(box.cell(f)), 1u)] = v;
            });
    }
    __syncthreads();
    auto cell_end = [&](uint32_t r) { return kLocal ? cur[r] : __ldcg(cur + r); };
    for (uint32_t r = tid; r < cells; r += T) {
        a.csr_start[so + r] = sh.cand0 + (r ? cell_end(r - 1) : 0u);   // read by other units' face cells
        if (kLocal) {
            a.stage_word[oo + r] = l_word[r];
            a.stage_lut[oo + r] = kRandom ? (uint32_t)l_key[r] : l_idx[r];
        } else if (kRandom) {
            a.stage_lut[oo + r] = (uint32_t)__ldcg(a.best + so + r);
        }
    }
    if (!a.spread) weighted_emit<kLocal, kB, Pre>(a, sh, box, l_word, cur, cells, oo, ws);
}

// Pass B and the emit of one unit.  kLocal: the cells' keys, sums and words
// are in shared memory (`pool`); otherwise (more cells than fit, or colour
// sums beyond 16 bits) in the staging arrays and the level's scratch, reached
// by reductions.  keep: the cells of this thread's first four candidates.
// Returns false (every thread alike) when a local unit has to be redone.
template <int T, int kColor, bool kRandom, int kB, bool kLocal, bool kOther, class Pre>
__device__ __forceinline__ bool unit_cells(const UnitLevelArgs& a, BlockShared& sh, const Box<kB, Pre>& box, uint32_t* pool,
                                           uint32_t ui, uint32_t cells, const int (&keep)[4], uint32_t claim,
                                           uint32_t included, bool placed, WeightShared* ws) {
    constexpr bool averaged = kColor == 1 || kColor == 2, weighted = kColor == 3;
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const Unit& un = sh.un;
    // shared: [sums 8 B, dense 16 B][random keys 8 B | indices 4 B][words 4 B][weighted: candidates 4 B] per cell
    const bool dense = kOther && kLocal && averaged && dense_unit(un.cnt, cells);
    uint2* l_sum = reinterpret_cast<uint2*>(pool);
    uint4* l_wide = reinterpret_cast<uint4*>(pool);   // dense: r, g, b, candidates
    uint64_t* l_key = reinterpret_cast<uint64_t*>(l_sum + (averaged ? dense ? 2 * cells : cells : 0));
    uint32_t* l_idx = reinterpret_cast<uint32_t*>(l_key);
    uint32_t* l_word = kRandom ? reinterpret_cast<uint32_t*>(l_key + cells) : l_idx + cells;
    uint32_t* l_cnt = l_word + cells;
    if (!kLocal && !placed) {
        if (warp == 0) unit_place(a, sh, ui, cells);
        __syncthreads();
    }
    uint64_t so = 0, oo = 0;
    if (!kLocal) {
        if (sh.fail) return true;
        so = sh.off + sh.rank0;
        oo = sh.level_base + so;
    }
    for (uint32_t r = tid; r < cells; r += T) {
        if (kLocal) {
            if (dense) l_wide[r] = make_uint4(0, 0, 0, 0);
            else if (averaged) l_sum[r] = make_uint2(0, 0);
            if (weighted) l_cnt[r] = 0;
            if (kRandom) l_key[r] = ~0ull;
            else l_idx[r] = 0xFFFFFFFFu;
        } else {
            if (kRandom) a.best[so + r] = ~0ull;
            else a.stage_lut[oo + r] = 0xFFFFFFFFu;
            if (kColor == 1) a.stage_col[oo + r] = 0;
            if (kColor == 2) a.sum[so + r] = 0;
            if (weighted) a.csr_count[so + r] = 0;
        }
    }
    if (kOther && !kLocal && un.large) {   // the rest is k_large_cells' and k_large_emit's
        if (tid == 0) a.maps[un.map + large_state(un.b) + 2] = sh.cand0;
        return true;
    }
    if (tid == 0) {
        sh.next = 0;
        sh.redo = 0;
        sh.delta = 0;
    }
    __syncthreads();

    {
        const uint32_t cnt = un.cnt, base = un.base;
        const bool staged = un.staged;
        const uint32_t shift = staged ? 1u : kFieldBits - a.s;
        const uint64_t start = un.start;
        const uint32_t* src_word = (staged ? a.stage_word : a.leaf_word) + start;
        const uint32_t* src_lut = (staged ? a.stage_lut : a.leaf_lut) + start;
        uint32_t wide = 0;   // colour bits above 8
        auto add = [&](uint32_t rank, uint32_t idx, uint32_t c0, uint32_t c1) {
            if (kRandom) {
                const SubNode& nd = a.nodes[un.node];
                const unsigned long long key =
                    ((unsigned long long)rp_priority(a.seed, nd.level, nd.morton, idx) << 32) | idx;
                if (!kLocal) atomicMin(reinterpret_cast<unsigned long long*>(a.best + so + rank), key);
                else if (key < *(volatile uint64_t*)&l_key[rank])
                    atomicMin(reinterpret_cast<unsigned long long*>(l_key + rank), key);
            } else if (kLocal) {
                atomicMin(l_idx + rank, idx);
            } else {
                atomicMin(a.stage_lut + oo + rank, idx);
            }
            if (averaged) {
                if (dense) {
                    atomicAdd(&l_wide[rank].x, c0 & 0xFFFFu);
                    atomicAdd(&l_wide[rank].y, c0 >> 16);
                    atomicAdd(&l_wide[rank].z, c1);
                    atomicAdd(&l_wide[rank].w, 1u);
                    wide |= (c0 & 0xFF00FF00u) | (c1 & 0xFF00u);
                } else if (kLocal) {
                    // r | g << 16 and b | 1 << 20: exact while the cell has at
                    // most 257 candidates with colours of 8 bits (checked below)
                    atomicAdd(&l_sum[rank].x, c0);
                    atomicAdd(&l_sum[rank].y, c1 | (1u << 20));
                    wide |= (c0 & 0xFF00FF00u) | (c1 & 0xFF00u);
                } else {
                    atomicAdd(reinterpret_cast<unsigned long long*>(kColor == 1 ? a.stage_col + oo + rank
                                                                                : a.sum + so + rank),
                              (unsigned long long)encode_colors(c0 & 0xFFFFu, c0 >> 16, c1));
                }
            }
            if (weighted) atomicAdd(kLocal ? l_cnt + rank : a.csr_count + so + rank, 1u);
        };
        for (uint32_t k0 = tid, it = 0; k0 < cnt; k0 += 4 * T, it += 4) {
            uint32_t idx[4], c0[4], c1[4];
            int i[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const uint32_t k = k0 + j * T;
                i[j] = -1;
                idx[j] = c0[j] = c1[j] = 0;
                if (k < cnt) {
                    idx[j] = src_lut[k];
                    if (averaged) {
                        if (staged) {
                            const uint2 v = *reinterpret_cast<const uint2*>(a.stage_col + start + k);
                            c0[j] = v.x;
                            c1[j] = v.y;
                        } else {
                            // r, g, b at byte 12 of the leaf's 18-byte record
                            const uintptr_t ra = reinterpret_cast<uintptr_t>(a.leaf_rec + (start + k) * 18 + 12);
                            const uint32_t* q = reinterpret_cast<const uint32_t*>(ra & ~(uintptr_t)3);
                            const uint32_t cs = (uint32_t)(ra & 2) * 8;
                            const uint32_t q0 = q[0], q1 = q[1];
                            c0[j] = __funnelshift_r(q0, q1, cs);
                            c1[j] = (q1 >> cs) & 0xFFFFu;
                        }
                    }
                    if (it) {
                        const uint32_t w = src_word[k];
                        uint32_t f = w >> shift;
                        bool mine = true;
                        if ((w & kWordEdges) && unproven(a, w)) {
                            f = unproven_cell(a, un, k, w);
                            mine = f != ~0u;
                        }
                        if (mine) i[j] = (int)box.cell(f);
                    } else {
                        i[j] = keep[j];
                    }
                }
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                if (i[j] < 0) continue;
                const uint32_t rank = box.rank((uint32_t)i[j]);
                add(rank, idx[j], c0[j], c1[j]);
                if (it + j >= 32 || (claim >> (it + j)) & 1u) {
                    const uint32_t wd = base + box.coordinates((uint32_t)i[j]);
                    if (kLocal) l_word[rank] = wd;
                    else a.stage_word[oo + rank] = wd;
                }
            }
        }
        if (kOther && sh.foreign)
            foreign_points(a, un, sh.foreign, [&](uint32_t f, uint32_t idx, uint32_t c0, uint32_t c1) {
                const uint32_t i = box.cell(f), rank = box.rank(i);
                add(rank, idx, c0, c1);
                if (kLocal) l_word[rank] = base + box.coordinates(i);
                else a.stage_word[oo + rank] = base + box.coordinates(i);
            });
        if (kLocal && averaged && wide) sh.redo = 1;
        __syncthreads();
        // cells whose point lies beside a boundary take over how far up it matters
        if (sh.unsafe) {
            auto edge = [&](uint32_t rank, uint32_t idx, uint32_t w) {
                uint32_t best;
                if (kLocal) best = kRandom ? (uint32_t)l_key[rank] : l_idx[rank];
                else best = kRandom ? (uint32_t)__ldcg(a.best + so + rank) : __ldcg(a.stage_lut + oo + rank);
                if (best != idx) return;
                if (kLocal) l_word[rank] |= w & kWordEdges;
                else a.stage_word[oo + rank] |= w & kWordEdges;
            };
            for (uint32_t k = tid; k < cnt; k += T) {
                const uint32_t w = src_word[k];
                if (!(w & kWordEdges)) continue;
                const uint32_t idx = src_lut[k], f = unproven(a, w) ? unproven_cell(a, un, k, w) : w >> shift;
                if (f != ~0u) edge(box.rank(box.cell(f)), idx, w);
            }
            if (kOther && sh.foreign)
                foreign_points(a, un, sh.foreign, [&](uint32_t f, uint32_t idx, uint32_t, uint32_t) {
                    edge(box.rank(box.cell(f)), idx, f);
                });
        }
    }
    // ---- the sums as the packed words of the reference; a count field that
    // overflowed shows as a sum of counts short of the unit's candidates
    if (kLocal) {
        if (dense) {
            // (the packed words go where the reads below expect them, over sums
            // of lower ranks, which are read first)
            for (uint32_t r0 = 0; r0 < cells; r0 += T) {
                const uint32_t r = r0 + tid;
                const uint4 v = r < cells ? l_wide[r] : make_uint4(0, 0, 0, 0);
                __syncthreads();
                if (r < cells)
                    *reinterpret_cast<uint64_t*>(l_sum + r) =
                        ((uint64_t)v.x << 46) + ((uint64_t)v.y << 28) + ((uint64_t)v.z << 10) + v.w;
            }
        } else if (averaged) {
            int32_t d = -(int32_t)included;
            bool bad = false;
            for (uint32_t r = tid; r < cells; r += T) {
                const uint2 v = l_sum[r];
                const uint32_t n = v.y >> 20;
                d += (int32_t)n;
                bad = bad || n > 257;
                *reinterpret_cast<uint64_t*>(l_sum + r) = ((uint64_t)(v.x & 0xFFFFu) << 46) +
                                                          ((uint64_t)(v.x >> 16) << 28) +
                                                          ((uint64_t)(v.y & 0xFFFFFu) << 10) + n;
            }
            d = __reduce_add_sync(0xffffffffu, d);
            if (lane == 0) atomicAdd(&sh.delta, d);
            if (bad) sh.redo = 1;
        }
        if (warp == 0) unit_place(a, sh, ui, cells);
        __syncthreads();
        if (averaged && (sh.redo || sh.delta)) return false;
        if (sh.fail) return true;
        so = sh.off + sh.rank0;
        oo = sh.level_base + so;
    } else {
        __syncthreads();
    }
    // ---- emit
    const uint64_t* l_packed = reinterpret_cast<const uint64_t*>(l_sum);
    const uint64_t* g_packed = a.sum + so;
    const uint32_t m0 = box.m0(), open = un.open;
    if constexpr (weighted) {
        unit_weighted<T, kRandom, kB, kLocal, kOther, Pre>(a, sh, box, l_key, l_word, l_cnt, cells, keep, so, oo, *ws);
    } else {
        for (uint32_t r0 = warp * 32; r0 < cells; r0 += T) {
            const uint32_t r = r0 + lane;
            bool face = false;
            uint32_t w = 0;
            if (r < cells) {
                if (kLocal) w = l_word[r];
                else if (kColor == 2) w = a.stage_word[oo + r];
                if (kLocal) {
                    a.stage_word[oo + r] = w;
                    a.stage_lut[oo + r] = kRandom ? (uint32_t)l_key[r] : l_idx[r];
                } else if (kRandom) {
                    a.stage_lut[oo + r] = (uint32_t)__ldcg(a.best + so + r);
                }
                if (kColor == 2 && a.spread) {
                    if (kLocal) a.sum[so + r] = l_packed[r];
                    continue;
                }
                uint64_t e = 0;
                if (kColor == 1) e = kLocal ? l_packed[r] : __ldcg(a.stage_col + oo + r);
                if (kColor == 2) {
                    const uint32_t x = w & m0, y = (w >> kFieldBits) & m0, z = (w >> (2 * kFieldBits)) & m0;
                    face = (faces_of(x, y, z, m0) & open) != 0;
                    e = box.sum27(x, y, z, [&](uint32_t q) { return kLocal ? l_packed[q] : __ldcg(g_packed + q); });
                }
                if (averaged) {
                    if (!face) {
                        uint16_t cr, cg, cb;
                        decode_colors(e, cr, cg, cb);
                        e = pack_colour(cr, cg, cb);
                    }
                    a.stage_col[oo + r] = e;
                }
            }
            if (kColor == 2 && !a.spread)
                append_faces(a, un.node, sh.off, sh.rank0 + r, w,
                             !face ? 0ull : kLocal ? l_packed[r] : __ldcg(g_packed + r), face);
        }
    }
    return true;
}

// unit_cells on global memory out of line, for blocks of 1024 threads, which
// seldom need it: inlined, its registers weigh on the other variant's (level
// 4 of the 119.7M-point build 1.34 -> 1.27 ms; two blocks per SM, which
// need it often, lose by it: level 1 0.84 -> 1.13 ms).
template <int T, int kColor, bool kRandom, int kB, bool kOther, class Pre>
__device__ __noinline__ void unit_cells_global(const UnitLevelArgs& a, BlockShared& sh, const uint32_t* bm,
                                               const Pre* pre, uint32_t b, uint32_t ui, uint32_t cells, int4 keep4,
                                               uint32_t claim, uint32_t included, bool placed) {
    const int keep[4] = {keep4.x, keep4.y, keep4.z, keep4.w};
    const Box<kB, Pre> box{bm, pre, b};
    unit_cells<T, kColor, kRandom, kB, false, kOther, Pre>(a, sh, box, nullptr, ui, cells, keep, claim, included,
                                                             placed, nullptr);
}

// One unit: pass A, ranks, then its cells.  kOther: points of other units may
// have their cells here, or a cell hold very many candidates.
template <int T, int kColor, bool kRandom, int kB, bool kOther, class Pre>
__device__ __forceinline__ void unit_run(const UnitLevelArgs& a, BlockShared& sh, uint32_t* bm, uint32_t ui,
                                         WeightShared* ws) {
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const Unit& un = sh.un;
    const uint32_t b = kB ? (uint32_t)kB : un.b;
    const uint32_t W = bitmap_words(b);
    // one word past the bitmap is read; both areas in steps of 16 bytes
    Pre* pre = reinterpret_cast<Pre*>(bm + ((W + 4) & ~3u));
    uint32_t* pool = bm + ((W + 4) & ~3u) + ((W * (uint32_t)sizeof(Pre) / 4 + 4) & ~3u);
    const Box<kB, Pre> box{bm, pre, b};
    for (uint32_t i = tid; i < (W + 4) / 4; i += T) reinterpret_cast<uint4*>(bm)[i] = make_uint4(0, 0, 0, 0);
    if (un.first && warp == T / 32 - 1) {
        // the node's place in the level's scratch and in the staging arrays
        const SubNode& nd = a.nodes[un.node];
        uint32_t n = 0;
        if (lane < nd.nchild) {
            const bool st = (nd.child_kind >> lane) & 1u;
            n = st ? a.out_points[(uint32_t)nd.child_start[lane]] : nd.child_count[lane];
        }
        uint64_t p = n;
        for (int o = 4; o >= 1; o >>= 1) p += __shfl_xor_sync(0xffffffffu, p, o);
        if (lane == 0) {
            const uint64_t off =
                atomicAdd(reinterpret_cast<unsigned long long*>(a.level_used + a.level), (unsigned long long)p);
            const bool over = off + p > a.scratch_cap || sh.level_base + off + p > a.stage_cap || p >> 32;
            if (over) atomicOr(a.err, kErrCapacity);
            store_release(&a.node_state[un.node].off1, over ? ~0ull : off + 1);
        }
    }
    __syncthreads();

    // ---- pass A: occupancy.  The thread whose candidate marks a cell
    // first also writes the cell's word in pass B: its rounds are kept as
    // bits of `claim` (rounds past 32 write it always).
    uint32_t claim = 0, included = 0;
    int keep[4] = {-1, -1, -1, -1};
    {
        const uint32_t cnt = un.cnt;
        const uint32_t shift = un.staged ? 1u : kFieldBits - a.s;
        const uint32_t* src_word = (un.staged ? a.stage_word : a.leaf_word) + un.start;
        bool beside = false;   // a candidate lies beside a boundary between cells
        if (kOther && un.large) {
            const uint32_t* map = a.maps + un.map;
            for (uint32_t i = tid; i < W; i += T) bm[i] = map[i];
            if (tid == 0) included = map[large_state(b)];
        }
        for (uint32_t k0 = kOther && un.large ? cnt : tid, it = 0; k0 < cnt; k0 += 4 * T, it += 4) {
            uint32_t w[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const uint32_t k = k0 + j * T;
                w[j] = k < cnt ? src_word[k] : 0u;
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const uint32_t k = k0 + j * T;
                if (k >= cnt) break;
                uint32_t f = w[j] >> shift;
                if (w[j] & kWordEdges) {
                    beside = true;
                    if (unproven(a, w[j])) {
                        f = unproven_cell(a, un, k, w[j]);
                        if (f == ~0u) continue;
                    }
                }
                const uint32_t i = box.cell(f);
                ++included;
                if (it == 0) keep[j] = (int)i;
                const uint32_t bit = 1u << (i & 31);
                uint32_t old = *(volatile uint32_t*)&bm[i >> 5];
                if (!(old & bit)) old = atomicOr(&bm[i >> 5], bit);
                if (!(old & bit) && it + j < 32) claim |= 1u << (it + j);
            }
        }
        if (kOther && sh.foreign && !un.large) {
            foreign_points(a, un, sh.foreign, [&](uint32_t f, uint32_t, uint32_t, uint32_t) {
                const uint32_t i = box.cell(f);
                ++included;
                beside = beside || (f & kWordEdges);
                atomicOr(&bm[i >> 5], 1u << (i & 31));
            });
        }
        if (beside) sh.unsafe = 1;
        if (kColor == 3) {
            const uint32_t n = __reduce_add_sync(0xffffffffu, included);
            if (lane == 0) atomicAdd(&sh.included, n);
        }
    }
    __syncthreads();

    // ---- ranks: a thread scans kP consecutive words
    constexpr uint32_t kP = kB == 6 ? 16 : kB == 5 ? 2 : 1;
    uint32_t sum = 0, c[kP];
    const bool scans = tid * kP < W;
    if (scans) {
#pragma unroll
        for (uint32_t q = 0; q < kP; ++q) {
            c[q] = sum;
            sum += __popc(bm[tid * kP + q]);
        }
    }
    uint32_t incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= (uint32_t)o) incl += y;
    }
    if (lane == 31) sh.warp[warp] = incl;
    __syncthreads();
    uint32_t wi = lane < T / 32 ? sh.warp[lane] : 0u;
    const uint32_t own = __shfl_sync(0xffffffffu, wi, warp);
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, wi, o);
        if (lane >= (uint32_t)o) wi += y;
    }
    const uint32_t cells = __shfl_sync(0xffffffffu, wi, 31);
    const uint32_t run = __shfl_sync(0xffffffffu, wi, warp) - own + incl - sum;
    if (tid == 0)
        store_release(&a.unit_state[ui], ((uint64_t)(kColor == 3 ? sh.included : 0u) << 32) | (cells + 1));
    if (scans) {
        if (kP == 1) {
            pre[tid] = (Pre)run;
        } else if (sizeof(Pre) == 4) {
#pragma unroll
            for (uint32_t q = 0; q < kP; ++q) pre[tid * kP + q] = (Pre)(run + c[q]);
        } else {
#pragma unroll
            for (uint32_t q = 0; q < kP; q += 2)
                reinterpret_cast<uint32_t*>(pre)[(tid * kP + q) / 2] =
                    ((run + c[q]) & 0xFFFFu) | ((run + c[q + (kP > 1)]) << 16);
        }
    }
    if ((kColor >= 2 && a.spread) || (kOther && un.large)) {
        __syncthreads();
        uint32_t* map = a.maps + un.map;
        for (uint32_t i = tid; i < W; i += T) {
            map[i] = bm[i];
            map[W + 4 + i] = pre[i];
        }
        if (tid == 0) map[W] = 0;
    }
    // (unit_cells starts with a barrier after it cleared the cells)
    const uint32_t room = a.smem_words * 4 - (uint32_t)((pool - bm) * 4);
    bool placed = false;
    const uint32_t dense_bytes = kOther && (kColor == 1 || kColor == 2) && dense_unit(un.cnt, cells) ? 8u : 0u;
    if (sizeof(Pre) == 2 && cells * (cell_bytes(kColor, kRandom) + dense_bytes) <= room && !(kOther && un.large)) {
        if (unit_cells<T, kColor, kRandom, kB, true, kOther, Pre>(a, sh, box, pool, ui, cells, keep, claim, included, false, ws))
            return;
        placed = true;
        __syncthreads();
    }
    if constexpr (T == 1024)
        unit_cells_global<T, kColor, kRandom, kB, kOther, Pre>(a, sh, bm, pre, b, ui, cells,
                                                       make_int4(keep[0], keep[1], keep[2], keep[3]), claim, included,
                                                       placed);
    else
        unit_cells<T, kColor, kRandom, kB, false, kOther, Pre>(a, sh, box, pool, ui, cells, keep, claim, included, placed,
                                                                 ws);
}

// Units of other kinds than the level's frequent ones (among them large leaves
// and those with points from other units), out of line, so that
// their registers do not weigh on those (see launch_units).
template <int T, int kColor, bool kRandom>
__device__ __noinline__ void unit_run_other(const UnitLevelArgs& a, BlockShared& sh, uint32_t* bm, uint32_t ui,
                                            WeightShared* ws) {
    if (sh.un.b == 6) unit_run<T, kColor, kRandom, 6, true, uint32_t>(a, sh, bm, ui, ws);
    else if (sh.un.b == 5) unit_run<T, kColor, kRandom, 5, true, uint16_t>(a, sh, bm, ui, ws);
    else unit_run<T, kColor, kRandom, 0, true, uint16_t>(a, sh, bm, ui, ws);
}

#if OC_UNITS_PART == 0
// The level's points whose cell lies outside their unit, as a segment per unit
// (or chunk of one) and octant they belong to.  Reads the words of all
// candidates, for builds that were found to have such points.
constexpr int kForeignThreads = 256;

__global__ void __launch_bounds__(kForeignThreads) k_foreign(const __grid_constant__ UnitLevelArgs a, uint32_t chunks,
                                                             uint32_t colour) {
    __shared__ uint32_t s_count[8], s_at[8], s_stop;
    constexpr uint32_t T = kForeignThreads;
    const uint32_t tid = threadIdx.x;
    if (tid == 0) s_stop = *(volatile uint32_t*)a.err;
    __syncthreads();
    if (s_stop) return;
    for (uint32_t item = blockIdx.x; item < a.n_units * chunks; item += gridDim.x) {
        const Unit un = load_unit(a, item / chunks);
        const uint32_t per = un.cnt / chunks + 1, first = min(item % chunks * per, un.cnt), end = min(first + per, un.cnt);
        uint32_t* word = (un.staged ? a.stage_word : a.leaf_word) + un.start;
        const uint32_t* lut = (un.staged ? a.stage_lut : a.leaf_lut) + un.start;
        auto points = [&](auto&& get) {
            for (uint32_t k0 = first + tid; k0 < end; k0 += 4 * T) {
                uint32_t w[4];
#pragma unroll
                for (uint32_t j = 0; j < 4; ++j) w[j] = k0 + j * T < end ? word[k0 + j * T] : 0u;
#pragma unroll
                for (uint32_t j = 0; j < 4; ++j) {
                    if (!unproven(a, w[j])) continue;
                    const uint32_t k = k0 + j * T, f = resolved_word(a, un, word + k, w[j], lut[k]), h = a.s - 1;
                    if (!(f & kWordForeign)) continue;
                    const uint32_t x = f & 127, y = (f >> kFieldBits) & 127, z = (f >> (2 * kFieldBits)) & 127;
                    get(k, f, ((x >> h) << 2) | ((y >> h) << 1) | (z >> h));
                }
            }
        };
        if (tid < 8) s_count[tid] = 0;
        __syncthreads();
        points([&](uint32_t, uint32_t, uint32_t o) { atomicAdd(&s_count[o], 1u); });
        __syncthreads();
        if (tid < 8 && s_count[tid]) {
            const uint32_t n = s_count[tid], at = atomicAdd(a.foreign_used, n + 1);
            if ((uint64_t)at + n + 1 > a.foreign_cap) {
                atomicOr(a.err, kErrForeign);   // no room: the kernels of whole nodes
                s_at[tid] = ~0u;
            } else {
                a.foreign[at] = make_uint4(atomicExch(&a.foreign_head[un.node * 8 + tid], at + 1), n, 0, 0);
                s_at[tid] = at + 1;
            }
        }
        const bool any = __syncthreads_or(tid < 8 && s_count[tid]);
        if (any)
            points([&](uint32_t k, uint32_t f, uint32_t o) {
                if (s_at[o] == ~0u) return;
                uint32_t c0 = 0, c1 = 0;
                if (colour && un.staged) {
                    const uint2 v = *reinterpret_cast<const uint2*>(a.stage_col + un.start + k);
                    c0 = v.x;
                    c1 = v.y;
                } else if (colour) {
                    const uint16_t* v = reinterpret_cast<const uint16_t*>(a.leaf_rec + (un.start + k) * 18 + 12);
                    c0 = v[0] | ((uint32_t)v[1] << 16);
                    c1 = v[2];
                }
                a.foreign[atomicAdd(&s_at[o], 1u)] = make_uint4(f, lut[k], c0, c1);
            });
        __syncthreads();
    }
}
#endif

// kColor: 0 raw colour, 1 intra-cell, 2 inter-cell, 3 distance-weighted.  An
// inter-cell or weighted colour whose neighbourhood reaches into other units keeps its sum and goes to its
// node's face list (k_faces).
// kHalf: units of half the side (parts of split children, or a grid of 64) are frequent too.
template <int T, int kColor, bool kRandom, bool kHalf>
__global__ void __launch_bounds__(T, unit_blocks(T)) k_units(const __grid_constant__ UnitLevelArgs a) {
    extern __shared__ __align__(16) uint32_t dyn[];
    __shared__ BlockShared sh;
    const uint32_t tid = threadIdx.x;
    if (tid == 0) {
        uint64_t b = 0;
        for (uint32_t l = 1; l < a.level; ++l) b += a.level_used[l];
        sh.level_base = b;
        sh.stop = *(volatile uint32_t*)a.err;
    }
    __syncthreads();
    // after an error the tables of the levels below may not agree with each
    // other: nothing is read by them (a unit that gave up leaves cells without
    // points, and octants whose ends lie before their starts)
    if (sh.stop) return;
    for (;;) {
        __syncthreads();   // the previous unit is done with the shared state
        if (tid == 0) {
            const uint32_t u = atomicAdd(a.ticket, 1u);
            sh.unit = u;
            sh.unsafe = 0;
            sh.included = 0;
            if (u < a.n_units) {
                sh.un = load_unit(a, u);
                sh.foreign = a.foreign_head ? a.foreign_head[sh.un.node * 8 + sh.un.octant] : 0u;
            }
        }
        __syncthreads();
        const uint32_t ui = sh.unit;
        if (ui >= a.n_units) break;
        if (kColor != 3 && tid == T - 33 && a.n_units - ui > gridDim.x) prefetch_unit<kColor>(a, ui + gridDim.x);
        // (the weighted lists follow the pool)
        WeightShared* ws = reinterpret_cast<WeightShared*>(dyn + a.smem_words);
        if (sh.foreign || sh.un.large) unit_run_other<T, kColor, kRandom>(a, sh, dyn, ui, ws);
        else if (sh.un.b == 6 && sh.un.cnt <= 65535) unit_run<T, kColor, kRandom, 6, false, uint16_t>(a, sh, dyn, ui, ws);
        else if (kHalf && sh.un.b == 5 && sh.un.cnt <= 32768) unit_run<T, kColor, kRandom, 5, false, uint16_t>(a, sh, dyn, ui, ws);
        else unit_run_other<T, kColor, kRandom>(a, sh, dyn, ui, ws);
    }
}

// Leaves of many points (dense spots of a scan, coarse counting grids) would keep
// one block busy for milliseconds: `slices` blocks share each of them.  Before
// the level's units k_large_mark marks their cells in the bitmaps of their maps;
// their units (k_units) give the cells ranks and places and clear them; then
// k_large_cells adds the candidates to the cells by reductions in L2, and
// k_large_emit makes colours.  In distance weighting k_large_scan and
// k_large_scatter group the candidates by cell in between.
// Builds of 20M points, 16M of them in 16^3 cells of one leaf: first point 54.9
// -> 7.6 ms, inter-cell 93.7 -> 8.4, weighted 175 -> 32; 10M points of terrain
// on a counting grid of 8 (927,000 in a leaf): inter-cell 7.7 -> 1.0.
constexpr int kLargeThreads = 512;

// A block's share of a large leaf: the unit, its box over the map in global
// memory, and its part of n items.
struct LargePart {
    Unit un;
    uint32_t ui, slice, stop;
    __device__ __forceinline__ uint32_t first(uint32_t n, uint32_t slices) const {
        return (uint32_t)((uint64_t)n * slice / slices);
    }
    __device__ __forceinline__ uint32_t end(uint32_t n, uint32_t slices) const {
        return (uint32_t)((uint64_t)n * (slice + 1) / slices);
    }
};

__device__ __forceinline__ void load_large(const UnitLevelArgs& a, uint32_t slices, LargePart& s) {
    if (threadIdx.x == 0) {
        s.stop = *(volatile uint32_t*)a.err;
        s.ui = a.large[blockIdx.x / slices];
        s.slice = blockIdx.x % slices;
        if (!s.stop) s.un = load_unit(a, s.ui);
    }
    __syncthreads();
}

// The unit's first cell in the level's scratch.
__device__ __forceinline__ uint64_t large_cells_at(const UnitLevelArgs& a, const LargePart& s) {
    return a.node_state[s.un.node].off1 - 1 + a.unit_rank[s.ui];
}

__device__ __forceinline__ uint64_t level_base_of(const UnitLevelArgs& a) {
    uint64_t b = 0;
    for (uint32_t l = 1; l < a.level; ++l) b += a.level_used[l];
    return b;
}

// Calls get(cell in the box, word, position) for the part's own candidates.
template <class Get>
__device__ __forceinline__ void large_candidates(const UnitLevelArgs& a, const LargePart& s, uint32_t slices,
                                                 const Box<0, uint32_t>& box, Get&& get) {
    const uint32_t* src_word = a.leaf_word + s.un.start;
    const uint32_t first = s.first(s.un.cnt, slices), end = s.end(s.un.cnt, slices);
    for (uint32_t k0 = first + threadIdx.x; k0 < end; k0 += 4 * kLargeThreads) {
        uint32_t w[4];
#pragma unroll
        for (uint32_t j = 0; j < 4; ++j) w[j] = k0 + j * kLargeThreads < end ? src_word[k0 + j * kLargeThreads] : 0u;
#pragma unroll
        for (uint32_t j = 0; j < 4; ++j) {
            const uint32_t k = k0 + j * kLargeThreads;
            if (k >= end) break;
            uint32_t f = w[j] >> (kFieldBits - a.s);
            if ((w[j] & kWordEdges) && unproven(a, w[j])) {
                f = unproven_cell(a, s.un, k, w[j]);
                if (f == ~0u) continue;
            }
            get(box.cell(f), w[j], k);
        }
    }
}

// Points of other units whose cells lie in the leaf's (the first slice takes them).
__device__ __forceinline__ uint32_t large_foreign(const UnitLevelArgs& a, const LargePart& s) {
    return a.foreign_head && s.slice == 0 ? a.foreign_head[s.un.node * 8 + s.un.octant] : 0u;
}

__global__ void __launch_bounds__(kLargeThreads) k_large_mark(const __grid_constant__ UnitLevelArgs a, uint32_t slices) {
    __shared__ LargePart s;
    __shared__ __align__(16) uint32_t bm[bitmap_words(6)];
    load_large(a, slices, s);
    if (s.stop) return;
    const uint32_t W = bitmap_words(s.un.b);
    const Box<0, uint32_t> box{bm, nullptr, s.un.b};
    for (uint32_t i = threadIdx.x; i < W; i += kLargeThreads) bm[i] = 0;
    __syncthreads();
    uint32_t included = 0;
    bool beside = false;
    auto mark = [&](uint32_t i, uint32_t w) {
        ++included;
        beside = beside || (w & kWordEdges);
        const uint32_t bit = 1u << (i & 31);
        if (!(*(volatile uint32_t*)&bm[i >> 5] & bit)) atomicOr(&bm[i >> 5], bit);
    };
    large_candidates(a, s, slices, box, [&](uint32_t i, uint32_t w, uint32_t) { mark(i, w); });
    foreign_points(a, s.un, large_foreign(a, s), [&](uint32_t f, uint32_t, uint32_t, uint32_t) { mark(box.cell(f), f); });
    uint32_t* map = a.maps + s.un.map;
    const uint32_t n = __reduce_add_sync(0xffffffffu, included);
    if ((threadIdx.x & 31) == 0) atomicAdd(map + large_state(s.un.b), n);
    if (beside) map[large_state(s.un.b) + 1] = 1;
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < W; i += kLargeThreads)
        if (bm[i]) atomicOr(map + i, bm[i]);
}

template <int kColor, bool kRandom>
__global__ void __launch_bounds__(kLargeThreads) k_large_cells(const __grid_constant__ UnitLevelArgs a, uint32_t slices) {
    __shared__ LargePart s;
    load_large(a, slices, s);
    if (s.stop) return;
    const Unit& un = s.un;
    const uint32_t* map = a.maps + un.map;
    const Box<0, uint32_t> box{map, map + bitmap_words(un.b) + 4, un.b};
    const uint64_t so = large_cells_at(a, s), oo = level_base_of(a) + so;
    const SubNode& nd = a.nodes[un.node];
    auto add = [&](uint32_t i, uint32_t idx, uint32_t c0, uint32_t c1) {
        const uint32_t rank = box.rank(i);
        if (kRandom)
            atomicMin(reinterpret_cast<unsigned long long*>(a.best + so + rank),
                      ((unsigned long long)rp_priority(a.seed, nd.level, nd.morton, idx) << 32) | idx);
        else
            atomicMin(a.stage_lut + oo + rank, idx);
        if (kColor == 1 || kColor == 2)
            atomicAdd(reinterpret_cast<unsigned long long*>(kColor == 1 ? a.stage_col + oo + rank : a.sum + so + rank),
                      (unsigned long long)encode_colors(c0 & 0xFFFFu, c0 >> 16, c1));
        if (kColor == 3) atomicAdd(a.csr_count + so + rank, 1u);
        a.stage_word[oo + rank] = un.base + box.coordinates(i);   // (the same by every candidate of the cell)
    };
    large_candidates(a, s, slices, box, [&](uint32_t i, uint32_t, uint32_t k) {
        uint32_t c0 = 0, c1 = 0;
        if (kColor == 1 || kColor == 2) {
            const uint16_t* q = reinterpret_cast<const uint16_t*>(a.leaf_rec + (un.start + k) * 18 + 12);
            c0 = q[0] | ((uint32_t)q[1] << 16);
            c1 = q[2];
        }
        add(i, a.leaf_lut[un.start + k], c0, c1);
    });
    foreign_points(a, un, large_foreign(a, s), [&](uint32_t f, uint32_t idx, uint32_t c0, uint32_t c1) {
        add(box.cell(f), idx, c0, c1);
    });
}

// Exclusive scan of the cells' candidates, in place: a block per leaf.
__global__ void __launch_bounds__(1024) k_large_scan(const __grid_constant__ UnitLevelArgs a) {
    __shared__ LargePart s;
    __shared__ uint32_t s_warp[32];
    load_large(a, 1, s);
    if (s.stop) return;
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, cells = (uint32_t)a.unit_state[s.ui] - 1u;
    uint32_t* count = a.csr_count + large_cells_at(a, s);
    uint32_t running = 0;
    for (uint32_t r0 = 0; r0 < cells; r0 += 1024) {
        const uint32_t r = r0 + tid, n = r < cells ? count[r] : 0u;
        uint32_t incl = n;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= (uint32_t)o) incl += y;
        }
        if (lane == 31) s_warp[warp] = incl;
        __syncthreads();
        uint32_t before = running, total = 0;
        for (uint32_t q = 0; q < 32; ++q) {
            before += q < warp ? s_warp[q] : 0u;
            total += s_warp[q];
        }
        if (r < cells) count[r] = before + incl - n;
        running += total;
        __syncthreads();
    }
}

__global__ void __launch_bounds__(kLargeThreads) k_large_scatter(const __grid_constant__ UnitLevelArgs a, uint32_t slices) {
    __shared__ LargePart s;
    load_large(a, slices, s);
    if (s.stop) return;
    const Unit& un = s.un;
    const uint32_t* map = a.maps + un.map;
    const Box<0, uint32_t> box{map, map + bitmap_words(un.b) + 4, un.b};
    uint32_t* cur = a.csr_count + large_cells_at(a, s);
    const uint64_t c0 = a.node_state[un.node].off1 - 1 + map[large_state(un.b) + 2];
    const SubNode& nd = a.nodes[un.node];
    large_candidates(a, s, slices, box, [&](uint32_t i, uint32_t, uint32_t k) {
        const uint16_t* q = reinterpret_cast<const uint16_t*>(a.leaf_rec + (un.start + k) * 18 + 12);
        float4 v = cell_units(a, nd, a.leaf_lut[un.start + k]);
        v.w = __uint_as_float((uint32_t)q[0] | ((uint32_t)q[1] << 8) | ((uint32_t)q[2] << 16));
        a.csr_pts[c0 + atomicAdd(cur + box.rank(i), 1u)] = v;
    });
    foreign_points(a, un, large_foreign(a, s), [&](uint32_t f, uint32_t idx, uint32_t rg, uint32_t bl) {
        float4 v = cell_units(a, nd, idx);
        v.w = __uint_as_float((rg & 0xFFu) | ((rg >> 8) & 0xFF00u) | (bl << 16));
        a.csr_pts[c0 + atomicAdd(cur + box.rank(box.cell(f)), 1u)] = v;
    });
}

// The cells' selected points, how far up they matter (kWordEdge), and colours.
template <int kColor, bool kRandom>
__global__ void __launch_bounds__(kLargeThreads) k_large_emit(const __grid_constant__ UnitLevelArgs a, uint32_t slices) {
    __shared__ LargePart s;
    load_large(a, slices, s);
    if (s.stop) return;
    const Unit& un = s.un;
    const uint32_t* map = a.maps + un.map;
    const Box<0, uint32_t> box{map, map + bitmap_words(un.b) + 4, un.b};
    const uint64_t so = large_cells_at(a, s), oo = level_base_of(a) + so;
    const uint32_t cells = (uint32_t)a.unit_state[s.ui] - 1u, first = s.first(cells, slices), end = s.end(cells, slices);
    if (map[large_state(un.b) + 1]) {
        // (the point that a cell keeps has one lane, and the words' other bits stay)
        auto edge = [&](uint32_t rank, uint32_t idx, uint32_t w) {
            const uint32_t best = kRandom ? (uint32_t)a.best[so + rank] : a.stage_lut[oo + rank];
            if (best == idx) atomicOr(a.stage_word + oo + rank, w & kWordEdges);
        };
        large_candidates(a, s, slices, box, [&](uint32_t i, uint32_t w, uint32_t k) {
            if (w & kWordEdges) edge(box.rank(i), a.leaf_lut[un.start + k], w);
        });
        foreign_points(a, un, large_foreign(a, s), [&](uint32_t f, uint32_t idx, uint32_t, uint32_t) {
            edge(box.rank(box.cell(f)), idx, f);
        });
    }
    const uint32_t rank0 = a.unit_rank[s.ui];
    if constexpr (kColor == 3) {
        const uint32_t cand0 = map[large_state(un.b) + 2];
        const uint32_t* cur = a.csr_count + so;
        for (uint32_t r = first + threadIdx.x; r < end; r += kLargeThreads) {
            a.csr_start[so + r] = cand0 + (r ? cur[r - 1] : 0u);
            if (kRandom) a.stage_lut[oo + r] = (uint32_t)a.best[so + r];
        }
        if (a.spread) return;
        __shared__ BlockShared sh;
        __shared__ WeightShared ws;
        if (threadIdx.x == 0) {
            sh.un = un;
            sh.off = a.node_state[un.node].off1 - 1;
            sh.cand0 = cand0;
            sh.rank0 = rank0;
            sh.next = first;
        }
        __syncthreads();
        weighted_emit<false, 0, uint32_t>(a, sh, box, nullptr, cur, end, oo, ws);
    } else {
        const uint32_t lane = threadIdx.x & 31, m0 = box.m0();
        for (uint32_t r0 = first + (threadIdx.x & ~31u); r0 < end; r0 += kLargeThreads) {
            const uint32_t r = r0 + lane;
            bool face = false;
            uint32_t w = 0;
            uint64_t own = 0;
            if (r < end) {
                if (kRandom) a.stage_lut[oo + r] = (uint32_t)a.best[so + r];
                uint64_t e = 0;
                if (kColor == 1) e = a.stage_col[oo + r];
                if (kColor == 2 && !a.spread) {
                    w = a.stage_word[oo + r];
                    const uint32_t x = w & m0, y = (w >> kFieldBits) & m0, z = (w >> (2 * kFieldBits)) & m0;
                    face = (faces_of(x, y, z, m0) & un.open) != 0;
                    own = a.sum[so + r];
                    e = box.sum27(x, y, z, [&](uint32_t q) { return a.sum[so + q]; });
                }
                if (kColor == 1 || (kColor == 2 && !a.spread)) {
                    if (!face) {
                        uint16_t cr, cg, cb;
                        decode_colors(e, cr, cg, cb);
                        e = pack_colour(cr, cg, cb);
                    }
                    a.stage_col[oo + r] = e;
                }
            }
            if (kColor == 2 && !a.spread)
                append_faces(a, un.node, a.node_state[un.node].off1 - 1, rank0 + r, w, own, face);
        }
    }
}

// The neighbourhood of the cells on faces between the units of a node.  A
// block marks the node's face cells in bitmaps of the planes on both sides of
// every cut (a cell on several planes in the first axis's), lists their sums
// in the order of the bits, and adds to each cell of its slice of the list
// what the cells of other units around it hold.  About 5% of the cells are
// face cells: the planes of one node take 24 KB (72 KB where children are
// split) at S = 128.  Nine neighbours are looked up at a time, so that their
// loads overlap.
struct Planes {
    uint32_t s, cut;   // log2 of the grid and of the distance between cuts
    uint32_t np;       // planes per axis
    __device__ __forceinline__ int plane(uint32_t v) const {
        const uint32_t q = (1u << cut) - 1, r = v & q;
        if (r == 0 && v > 0) return (int)(2 * (v >> cut)) - 1;
        if (r == q && v + 1 < (1u << s)) return (int)(2 * (v >> cut));
        return -1;
    }
    // bit of a face cell with the planes of its coordinates
    __device__ __forceinline__ uint32_t index(uint32_t x, uint32_t y, uint32_t z, int px, int py, int pz) const {
        const uint32_t p = px >= 0 ? (uint32_t)px : py >= 0 ? np + (uint32_t)py : 2 * np + (uint32_t)max(pz, 0);
        const uint32_t u = px >= 0 ? y : x, v = px < 0 && py < 0 ? y : z;
        return (((p << s) | u) << s) | v;
    }
};

constexpr int kFaceThreads = 256;

template <int kColor>
__global__ void __launch_bounds__(kFaceThreads) k_faces(const __grid_constant__ UnitLevelArgs a, uint32_t slices,
                                                        uint32_t cut) {
    extern __shared__ __align__(16) uint32_t dyn[];
    __shared__ uint32_t s_warp[kFaceThreads / 32];
    constexpr uint32_t T = kFaceThreads;
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const Planes pl{a.s, cut, 2 * ((1u << (a.s - cut)) - 1)};
    const uint32_t W = max((3 * pl.np) << (2 * a.s) >> 5, 1u);
    uint32_t* bits = dyn;
    uint32_t* pre = dyn + W;
    if (*a.err) return;   // (set by earlier launches alone, as in k_spread)
    uint64_t level_base = 0;
    for (uint32_t l = 1; l < a.level; ++l) level_base += a.level_used[l];
    for (uint32_t item = blockIdx.x; item < a.n_nodes * slices; item += gridDim.x) {
        const uint32_t node = item / slices, slice = item % slices;
        const UnitNodeState st = a.node_state[node];
        const uint32_t F = st.off1 == ~0ull ? 0u : st.faces;
        if (slice * T / (kColor == 2 ? 1 : 8) >= F) continue;   // every thread alike
        const uint64_t off = st.off1 - 1;
        const uint32_t kind = a.nodes[node].child_kind;
        const uint2* list = a.faces + off;
        const uint64_t* list_sum = a.face_sum + off;
        uint64_t* table = a.sum + off;            // sums, or (weighted) ranks
        uint32_t* table_rank = a.csr_count + off;
        uint64_t* colour = a.stage_col + level_base + off;
        for (uint32_t i = tid; i < W; i += T) bits[i] = 0;
        __syncthreads();
        auto place = [&](uint32_t w) {
            const uint32_t x = w & 127, y = (w >> kFieldBits) & 127, z = (w >> (2 * kFieldBits)) & 127;
            return pl.index(x, y, z, pl.plane(x), pl.plane(y), pl.plane(z));
        };
        for (uint32_t f0 = tid; f0 < F; f0 += 4 * T) {
            uint32_t w[4];
#pragma unroll
            for (uint32_t j = 0; j < 4; ++j) w[j] = f0 + j * T < F ? list[f0 + j * T].y : 0u;
#pragma unroll
            for (uint32_t j = 0; j < 4; ++j) {
                const uint32_t i = place(w[j]);
                if (f0 + j * T < F) atomicOr(&bits[i >> 5], 1u << (i & 31));
            }
        }
        __syncthreads();
        const uint32_t per = (W + T - 1) / T, w0 = min(tid * per, W), w1 = min(w0 + per, W);
        uint32_t sum = 0;
        for (uint32_t q = w0; q < w1; ++q) sum += __popc(bits[q]);
        uint32_t incl = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= (uint32_t)o) incl += y;
        }
        if (lane == 31) s_warp[warp] = incl;
        __syncthreads();
        uint32_t run = incl - sum;
#pragma unroll
        for (uint32_t q = 0; q < T / 32; ++q) run += q < warp ? s_warp[q] : 0u;
        for (uint32_t q = w0; q < w1; ++q) {
            pre[q] = run;
            run += __popc(bits[q]);
        }
        __syncthreads();
        for (uint32_t f0 = tid; f0 < F; f0 += 4 * T) {
            uint2 v[4];
            uint64_t e[4];
#pragma unroll
            for (uint32_t j = 0; j < 4; ++j) {
                v[j] = f0 + j * T < F ? list[f0 + j * T] : make_uint2(0, 0);
                e[j] = kColor == 2 && f0 + j * T < F ? list_sum[f0 + j * T] : 0ull;
            }
#pragma unroll
            for (uint32_t j = 0; j < 4; ++j) {
                if (f0 + j * T >= F) break;
                const uint32_t i = place(v[j].y);
                const uint32_t at = pre[i >> 5] + __popc(bits[i >> 5] & ((1u << (i & 31)) - 1u));
                if (kColor == 2) table[at] = e[j];
                else table_rank[at] = v[j].x;
            }
        }
        __syncthreads();
        constexpr uint32_t kG = kColor == 2 ? 1 : 8;   // lanes per face cell
        const uint32_t g = tid % kG;
        const uint32_t node_cells = a.out_points[a.first_internal + node];
        // (whole warps, for the sums over lanes)
        for (uint32_t f0 = (slice * T + tid) / kG; f0 - tid / kG % (32 / kG) < F; f0 += slices * T / kG) {
            const uint32_t f = min(f0, F - 1);
            const uint2 v = list[f];
            uint64_t e = kColor == 2 ? colour[v.x] : 0ull;
            uint64_t ws[4] = {0, 0, 0, 0};
            const uint32_t c[3] = {v.y & 127, (v.y >> kFieldBits) & 127, (v.y >> (2 * kFieldBits)) & 127};
            const uint32_t h = a.s - 1, o = ((c[0] >> h) << 2) | ((c[1] >> h) << 1) | (c[2] >> h);
            const uint32_t ub = (kind >> (16 + o)) & 1u ? h - 1 : h;   // log2 side of the cell's unit
            if constexpr (kColor == 2) {
                int p[3][3];                 // planes of the coordinates - 1, 0, + 1
                uint32_t out = 0, far = 0;   // bits 3 * axis + step: outside the node, in another unit
#pragma unroll
                for (int k = 0; k < 3; ++k) {
#pragma unroll
                    for (int d = 0; d < 3; ++d) {
                        const uint32_t n = c[k] + d - 1;
                        p[k][d] = pl.plane(n);
                        out |= (n >> a.s ? 1u : 0u) << (3 * k + d);
                        far |= ((n ^ c[k]) >> ub ? 1u : 0u) << (3 * k + d);
                    }
                }
#pragma unroll
                for (int dz = 0; dz < 3; ++dz) {
                    uint32_t at[9];
#pragma unroll
                    for (int q = 0; q < 9; ++q) {
                        const int dx = q % 3, dy = q / 3;
                        const uint32_t m = (1u << dx) | (8u << dy) | (64u << dz);
                        at[q] = ~0u;
                        if (!(out & m) && (far & m)) {
                            const uint32_t i = pl.index(c[0] + dx - 1, c[1] + dy - 1, c[2] + dz - 1, p[0][dx],
                                                        p[1][dy], p[2][dz]);
                            const uint32_t bw = bits[i >> 5];
                            if ((bw >> (i & 31)) & 1u) at[q] = pre[i >> 5] + __popc(bw & ((1u << (i & 31)) - 1u));
                        }
                    }
#pragma unroll
                    for (int q = 0; q < 9; ++q)
                        if (at[q] != ~0u) e += table[at[q]];
                }
            } else {
                // eight lanes, each with every eighth neighbour
                for (uint32_t d = g; d < 27; d += kG) {
                    const uint32_t x = c[0] + d % 3 - 1, y = c[1] + d / 3 % 3 - 1, z = c[2] + d / 9 - 1;
                    if ((x | y | z) >> a.s) continue;
                    if ((((x ^ c[0]) | (y ^ c[1]) | (z ^ c[2])) >> ub) == 0) continue;
                    const uint32_t i = pl.index(x, y, z, pl.plane(x), pl.plane(y), pl.plane(z));
                    const uint32_t bw = bits[i >> 5];
                    if (!((bw >> (i & 31)) & 1u)) continue;
                    const uint32_t n = table_rank[pre[i >> 5] + __popc(bw & ((1u << (i & 31)) - 1u))];
                    const uint32_t end = n + 1 < node_cells ? a.csr_start[off + n + 1] : st.points;
                    for (uint32_t k = a.csr_start[off + n]; k < end; ++k) {
                        const float4 u = a.csr_pts[off + k];
                        const uint32_t col = __float_as_uint(u.w);
                        const uint32_t wq = weight_q(u.x, u.y, u.z, (int)c[0], (int)c[1], (int)c[2]);
                        ws[0] += (uint64_t)wq * (col & 0xFFu);
                        ws[1] += (uint64_t)wq * ((col >> 8) & 0xFFu);
                        ws[2] += (uint64_t)wq * (col >> 16);
                        ws[3] += wq;
                    }
                }
                __syncwarp();
            }
            if (kColor == 2) {
                uint16_t cr, cg, cb;
                decode_colors(e, cr, cg, cb);
                if (f0 < F) colour[v.x] = pack_colour(cr, cg, cb);
            } else {
#pragma unroll
                for (int q = 0; q < 4; ++q)
                    for (int o = kG / 2; o >= 1; o >>= 1) ws[q] += __shfl_xor_sync(0xffffffffu, ws[q], o);
                if (f0 < F && g == 0) {
                    const uint64_t* p = a.partial + list_sum[f] * 4;
                    const uint64_t sw = ws[3] + p[3];
                    colour[v.x] = pack_colour((uint16_t)weighted_mean(ws[0] + p[0], sw),
                                              (uint16_t)weighted_mean(ws[1] + p[1], sw),
                                              (uint16_t)weighted_mean(ws[2] + p[2], sw));
                }
            }
        }
        __syncthreads();   // the bitmaps are cleared for the next node
    }
}

// The colours of a level of few units (the top of the tree, where one unit's
// cells would keep one SM busy while others idle): `chunks` blocks per unit,
// each every chunks-th run of its cells.  Neighbours are looked up in the
// units' bitmaps in global memory, those of other units through the node's
// octant table, so that no cells are left over for k_faces.
// Bounded by the weights' instructions.  Root of the 25.8M-point weighted
// build (115,000 cells, 64 units of very unequal size): 1.27 -> 0.35 ms; levels
// 8 and 7 1.24 -> 0.54 and 1.15 -> 0.88 ms.
constexpr int kSpreadThreads = 256;

struct SpreadMap {
    const uint32_t* map;   // null: no such unit
    uint32_t b, rank;      // log2 side of its box, rank of its first cell in the node
};

__device__ __forceinline__ SpreadMap spread_map(const UnitLevelArgs& a, uint32_t node, uint32_t x, uint32_t y,
                                                uint32_t z) {
    const uint32_t h = a.s - 1, o = ((x >> h) << 2) | ((y >> h) << 1) | (z >> h);
    uint32_t u = a.oct_unit[node * 8 + o];
    SpreadMap m{nullptr, h, 0};
    if (u == ~0u) return m;
    if (u >> 31) {
        m.b = h - 1;
        u = (u & 0x7FFFFFFFu) +
            ((((x >> m.b) & 1) << 2) | (((y >> m.b) & 1) << 1) | ((z >> m.b) & 1));
    }
    m.map = a.maps + a.units[u].map;
    m.rank = a.unit_rank[u];
    return m;
}

// Occupied cells among the n at (x, y, z), (x + 1, y, z), ... of the unit's
// box, as bits, and the node rank of the first of them.
__device__ __forceinline__ uint32_t spread_row(const SpreadMap& m, uint32_t x, uint32_t y, uint32_t z, uint32_t n,
                                               uint32_t& rank) {
    if (!m.map) return 0;
    const uint32_t m0 = (1u << m.b) - 1u, i = (x & m0) | ((y & m0) << m.b) | ((z & m0) << (2 * m.b)), w = i >> 5;
    const uint32_t lo = m.map[w], t = __funnelshift_r(lo, m.map[w + 1], i) & ((1u << n) - 1u);
    if (t) rank = m.rank + m.map[(1u << (3 * m.b - 5)) + 4 + w] + __popc(lo & ((1u << (i & 31)) - 1u));
    return t;
}

template <int kColor>
__global__ void __launch_bounds__(kSpreadThreads) k_spread(const __grid_constant__ UnitLevelArgs a, uint32_t chunks) {
    constexpr uint32_t T = kSpreadThreads, kG = kColor == 3 ? kWeightLanes : 1;
    __shared__ uint2 s_rows[kColor == 3 ? T / kG : 1][18];
    const uint32_t tid = threadIdx.x, lane = tid & 31, s = lane % kG;
    const uint32_t ui = blockIdx.x / chunks, chunk = blockIdx.x % chunks;
    if (*a.err) return;
    const uint32_t cells = (uint32_t)a.unit_state[ui] - 1u;
    const UnitEntry en = a.units[ui];
    const UnitNodeState st = a.node_state[en.node];
    if (st.off1 == ~0ull || cells + 1 == 0 || chunk * (T / kG) >= cells) return;
    uint64_t level_base = 0;
    for (uint32_t l = 1; l < a.level; ++l) level_base += a.level_used[l];
    const uint64_t off = st.off1 - 1;
    const uint32_t rank0 = a.unit_rank[ui], node_cells = a.out_points[a.first_internal + en.node];
    const uint32_t* words = a.stage_word + level_base + off + rank0;
    uint64_t* colour = a.stage_col + level_base + off + rank0;
    const uint32_t S = 1u << a.s;
    const bool part = (en.flags >> 3) & 15;
    const SpreadMap own{a.maps + en.map, part ? a.s - 2 : a.s - 1, rank0};
    for (uint32_t f0 = chunk * (T / kG) + tid / kG; f0 - lane / kG < cells; f0 += chunks * (T / kG)) {
        const bool act = f0 < cells;
        const uint32_t w = words[min(f0, cells - 1)];
        const uint32_t x = w & 127, y = (w >> kFieldBits) & 127, z = (w >> (2 * kFieldBits)) & 127;
        // a row of up to three cells: those in the box of the cell's own x,
        // and one more across its side
        auto row = [&](uint32_t k, uint32_t (&t)[2], uint32_t (&rank)[2]) {
            const uint32_t yy = y + k % 3 - 1, zz = z + k / 3 - 1;
            t[0] = t[1] = 0;
            if (!act || k >= 9 || yy >= S || zz >= S) return;
            const bool inside = (((yy ^ y) | (zz ^ z)) >> own.b) == 0;
            const SpreadMap m = inside ? own : spread_map(a, en.node, x, yy, zz);
            const uint32_t q = (1u << m.b) - 1u, lx = x & q;
            const uint32_t xa = lx ? x - 1 : x, xb = lx < q ? x + 1 : x;
            t[0] = spread_row(m, xa, yy, zz, xb - xa + 1, rank[0]);
            const uint32_t side = lx ? x + 1 : x - 1;   // beyond the box when lx is its first or last cell
            if ((lx == 0 || lx == q) && side < S)
                t[1] = spread_row(spread_map(a, en.node, side, yy, zz), side, yy, zz, 1, rank[1]);
        };
        if constexpr (kColor == 2) {
            uint64_t e = 0;
#pragma unroll 3
            for (uint32_t k = 0; k < 9; ++k) {
                uint32_t t[2], rank[2];
                row(k, t, rank);
                const uint64_t* p = a.sum + off;
                if (t[0]) e += p[rank[0]];
                if (t[0] & (t[0] - 1)) e += p[rank[0] + 1];
                if (t[0] == 7) e += p[rank[0] + 2];
                if (t[1]) e += p[rank[1]];
            }
            uint16_t cr, cg, cb;
            decode_colors(e, cr, cg, cb);
            if (act) colour[f0] = pack_colour(cr, cg, cb);
        } else {
            uint2* rows = s_rows[tid / kG];
            constexpr uint32_t kR = (9 + kG - 1) / kG;
            uint32_t from[2 * kR], len[2 * kR], sum = 0;
#pragma unroll
            for (uint32_t q = 0; q < kR; ++q) {
                uint32_t t[2], rank[2];
                row(s + q * kG, t, rank);
#pragma unroll
                for (int d = 0; d < 2; ++d) {
                    from[2 * q + d] = len[2 * q + d] = 0;
                    if (t[d]) {
                        const uint32_t n = rank[d] + __popc(t[d]);
                        from[2 * q + d] = a.csr_start[off + rank[d]];
                        len[2 * q + d] = (n < node_cells ? a.csr_start[off + n] : st.points) - from[2 * q + d];
                    }
                    sum += len[2 * q + d];
                }
            }
            uint32_t incl = sum;
#pragma unroll
            for (uint32_t o = 1; o < kG; o <<= 1) {
                const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o, kG);
                if (s >= o) incl += v;
            }
            const uint32_t total = __shfl_sync(0xffffffffu, incl, kG - 1, kG);
            uint32_t run = incl - sum;
#pragma unroll
            for (uint32_t q = 0; q < 2 * kR; ++q) {
                const uint32_t slot = 2 * (s * (9 / kG) + min(s, 9 % kG)) + q;
                if (s + q / 2 * kG < 9) rows[slot] = make_uint2(run + len[q], from[q] - run);
                run += len[q];
            }
            __syncwarp();
            uint64_t sr = 0, sg = 0, sb = 0, sw = 0;
            const float cx = __fadd_rn((float)x, 0.5f), cy = __fadd_rn((float)y, 0.5f), cz = __fadd_rn((float)z, 0.5f);
            uint2 e = rows[0];
            const float4* pts = a.csr_pts + off;
            for (uint32_t p = s, k = 0; p < total; p += kG) {
                while (p >= e.x) e = rows[++k];
                const float4 v = pts[e.y + p];
                const uint32_t c = __float_as_uint(v.w);
                const uint32_t wq = weight_at(v.x, v.y, v.z, cx, cy, cz);
                sr += (uint64_t)wq * (c & 0xFFu);
                sg += (uint64_t)wq * ((c >> 8) & 0xFFu);
                sb += (uint64_t)wq * (c >> 16);
                sw += wq;
            }
#pragma unroll
            for (uint32_t o = kG / 2; o >= 1; o >>= 1) {
                sr += __shfl_xor_sync(0xffffffffu, sr, o);
                sg += __shfl_xor_sync(0xffffffffu, sg, o);
                sb += __shfl_xor_sync(0xffffffffu, sb, o);
                sw += __shfl_xor_sync(0xffffffffu, sw, o);
            }
            uint32_t c = 0;
            if (act && s < 3) c = weighted_mean(s == 0 ? sr : s == 1 ? sg : sb, sw);
            const uint32_t c1 = __shfl_sync(0xffffffffu, c, 1, kG), c2 = __shfl_sync(0xffffffffu, c, 2, kG);
            if (act && s == 0) colour[f0] = pack_colour((uint16_t)c, (uint16_t)c1, (uint16_t)c2);
            __syncwarp();   // the rows are written for the next cells
        }
    }
}

// Records of all internal nodes at their final positions (post-order after
// the n leaf records): output coordinates from the cloud point as in
// distribution, colours from the staging array (or, raw, the cloud point's).
// Bound by the reads of cloud points all over the cloud, 57 bytes of DRAM
// traffic per point for 24: 86 in all, at 5.3 TB/s (115M records 2.19 -> 1.88
// ms with coordinates in fixed point instead of float-float, which left more
// registers for loads; two or four gathers per lane in flight leave too few
// warps: 3.1 and 2.05 ms).
// A warp takes runs of 128 records; the node of its first record comes from a
// search over the nodes' first positions.
template <bool kF32, bool kAveraged>
__global__ void __launch_bounds__(256) k_place_units(const uint64_t* __restrict__ src_off,
                                                     const uint64_t* __restrict__ dst_off,
                                                     const uint32_t* __restrict__ count, uint32_t n_nodes, uint64_t n,
                                                     const uint64_t* __restrict__ total, OutParams op,
                                                     const __grid_constant__ FixedGrid fg,
                                                     const uint8_t* __restrict__ cloud, uint32_t stride,
                                                     const uint32_t* __restrict__ stage_lut,
                                                     const uint64_t* __restrict__ stage_col, uint8_t* __restrict__ rec,
                                                     uint32_t* err) {
    __shared__ __align__(16) uint8_t s_stage[8 * kStageBytes];
    constexpr uint32_t kRun = 128;
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint8_t* stage = s_stage + warp * kStageBytes;
    if (*err) return;   // levels may be without outputs: nothing was placed
    const uint64_t end = n + *total;
    const uint64_t step = (uint64_t)gridDim.x * 8 * kRun;
    for (uint64_t p0 = n + ((uint64_t)blockIdx.x * 8 + warp) * kRun; p0 < end; p0 += step) {
        uint32_t lo = 0, hi = n_nodes;   // last node with dst_off <= p0
        while (hi - lo > 1) {
            const uint32_t mid = (lo + hi) / 2;
            if (dst_off[mid] <= p0) lo = mid;
            else hi = mid;
        }
        uint32_t v = lo;
        for (uint32_t q = 0; q < kRun && p0 + q < end; q += 32) {
            const uint64_t p = p0 + q + lane;
            uint32_t nw[5] = {0, 0, 0, 0, 0};
            if (p < end) {
                while (p >= dst_off[v] + count[v] && v + 1 < n_nodes) ++v;
                const uint64_t s = src_off[v] + (p - dst_off[v]);
                const uint32_t idx = min(stage_lut[s], (uint32_t)n - 1u);   // a failed pass may leave any value
                uint32_t w[kF32 ? 4 : 7];
                gather_words<kF32, !kAveraged>(cloud + (uint64_t)idx * stride, w);
                fixed_out_coords<kF32>(w, fg, op.ax, nw);
                if (kAveraged) {
                    const uint2 e = *reinterpret_cast<const uint2*>(stage_col + s);
                    nw[3] = e.x;
                    nw[4] = e.y;
                } else {
                    const uint32_t col = w[kF32 ? 3 : 6];
                    nw[3] = (col & 0xFFu) | (((col >> 8) & 0xFFu) << 16);
                    nw[4] = (col >> 16) & 0xFFu;
                }
            }
            store_run(rec + (p0 + q) * 18, 0, (uint32_t)min((unsigned long long)32, (unsigned long long)(end - p0 - q)),
                      nw, stage);
        }
    }
}

// Resident blocks of a kernel per SM at a shared-memory size, queried once
// per device, kernel and size.
int blocks_per_sm(const void* kernel, int threads, size_t smem) {
    static std::mutex mu;
    static std::map<std::pair<std::pair<int, const void*>, size_t>, int> known;
    int dev = 0;
    cudaGetDevice(&dev);
    const auto key = std::make_pair(std::make_pair(dev, kernel), smem);
    std::lock_guard<std::mutex> g(mu);
    auto it = known.find(key);
    if (it != known.end()) return it->second;
    int n = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel, threads, smem) != cudaSuccess) {
        cudaGetLastError();
        n = 0;
    }
    n = std::max(n, 1);
    known[key] = n;
    return n;
}

// Shared memory of a unit block: an equal share of an SM's 227 KB, less the
// static part and the 1 KB the system takes per block.
template <int T, int kColor, bool kRandom, bool kHalf>
void launch_units_of(UnitLevelArgs a, int num_sms, cudaStream_t stream) {
    const size_t smem = (227 * 1024 / unit_blocks(T) - 1024 - sizeof(BlockShared)) & ~(size_t)127;
    a.smem_words = (uint32_t)((smem - (kColor == 3 ? sizeof(WeightShared) : 0)) / 4) & ~3u;
    auto kern = k_units<T, kColor, kRandom, kHalf>;
    allow_dynamic_smem(reinterpret_cast<const void*>(kern), smem);
    const uint64_t fit =
        (uint64_t)std::max(num_sms, 1) * blocks_per_sm(reinterpret_cast<const void*>(kern), T, smem);
    kern<<<(unsigned)std::min<uint64_t>(a.n_units, fit), T, smem, stream>>>(a);
}

// Blocks of 1024 where every unit has an SM of its own, and on levels of many
// units whose cells would mostly not fit in half an SM's shared memory
// (candidates x bytes per cell; a unit that does not fit works in global
// memory).  Levels 8 and 9 of the 25.8M-point random planes 106 -> 86 and
// 115 -> 68 us, level 5 (104 KB) 481 -> 453; 12.3M-point terrain, level 4
// (140 KB) 330 -> 278 us; but 119.7M points, level 3 (74 KB): 2.42 ms with two
// blocks, 2.82 with one.  With 1 to 3 units per SM two blocks are the better
// balance (level of 294 units: 135 us against 172).
//
// `half`: units of half the side are frequent.  Only the frequent kinds are in
// line in a kernel, and two blocks of 640 then have registers enough (with all
// kinds in line 640 threads gained nothing over 512; 704 and 768 gain less).
// 119.7M points, levels 2 and 3, 0.96 -> 0.87 and 2.31 -> 2.07 ms; 5.1M points
// 1.10 -> 1.03; 25.8M, level 4, 0.34 -> 0.30.  Both kinds in line everywhere:
// level 3 2.20; out of line where they are frequent: level 8 of 25.8M points
// 80 -> 106 us, weighted 0.51 -> 0.53 ms.
template <int kColor, bool kRandom>
void launch_units(const UnitLevelArgs& a, uint32_t mean_candidates, bool half, int num_sms, cudaStream_t stream) {
    if constexpr (kColor == 3) {
        if (half) launch_units_of<kWeightThreads, kColor, kRandom, true>(a, num_sms, stream);
        else launch_units_of<kWeightThreads, kColor, kRandom, false>(a, num_sms, stream);
    } else {
        const uint64_t sms = (uint64_t)std::max(num_sms, 1);
        const bool wide = a.n_units <= sms ||
                          (a.n_units >= 3 * sms && (uint64_t)mean_candidates * cell_bytes(kColor, kRandom) > 78 * 1024);
        if (wide) launch_units_of<1024, kColor, kRandom, false>(a, num_sms, stream);
        else if (half) launch_units_of<640, kColor, kRandom, true>(a, num_sms, stream);
        else launch_units_of<640, kColor, kRandom, false>(a, num_sms, stream);
    }
}

template <int kColor, bool kRandom>
int launch_large(const UnitLevelArgs& a, uint32_t slices, cudaStream_t stream) {
    const unsigned grid = a.n_large * slices;
    k_large_cells<kColor, kRandom><<<grid, kLargeThreads, 0, stream>>>(a, slices);
    if (kColor == 3) {
        k_large_scan<<<a.n_large, 1024, 0, stream>>>(a);
        k_large_scatter<<<grid, kLargeThreads, 0, stream>>>(a, slices);
    }
    k_large_emit<kColor, kRandom><<<grid, kLargeThreads, 0, stream>>>(a, slices);
    return kColor == 3 ? 5 : 3;
}

// Half-size units are frequent where children are split and on grids up to 64.
// Large leaves are shared by blocks of about 4096 candidates, up to eight per SM.
template <int kColor>
int launch_units_as(const UnitLevelArgs& a, bool random, uint32_t mean_candidates, bool any_split, int num_sms,
                    cudaStream_t stream) {
    const bool half = any_split || a.s <= 6;
    uint32_t slices = 1;
    if (a.n_large) {
        const uint64_t sms = (uint64_t)std::max(num_sms, 1);
        slices = (uint32_t)std::max<uint64_t>(1, std::min<uint64_t>(a.largest / 4096, (8 * sms + a.n_large - 1) / a.n_large));
        k_large_mark<<<a.n_large * slices, kLargeThreads, 0, stream>>>(a, slices);
    }
    if (random) launch_units<kColor, true>(a, mean_candidates, half, num_sms, stream);
    else launch_units<kColor, false>(a, mean_candidates, half, num_sms, stream);
    if (!a.n_large) return 1;
    return 1 + (random ? launch_large<kColor, true>(a, slices, stream) : launch_large<kColor, false>(a, slices, stream));
}

template <int kColor>
void launch_faces(const UnitLevelArgs& a, bool any_split, int num_sms, cudaStream_t stream) {
    const uint32_t cut = any_split ? a.s - 2 : a.s - 1;
    const uint32_t np = 2 * ((1u << (a.s - cut)) - 1);
    const size_t smem = (size_t)std::max((3 * np) << (2 * a.s) >> 5, 1u) * 8;
    auto kern = k_faces<kColor>;
    allow_dynamic_smem(reinterpret_cast<const void*>(kern), smem);
    const uint64_t fit = (uint64_t)std::max(num_sms, 1) *
                         blocks_per_sm(reinterpret_cast<const void*>(kern), kFaceThreads, smem);
    // a node's list is shared between up to 16 blocks (its length is not known
    // here: blocks without a part of it leave at once)
    uint32_t slices = 1;
    while (slices < 16 && (uint64_t)a.n_nodes * slices < 4 * fit) slices <<= 1;
    kern<<<(unsigned)std::min<uint64_t>((uint64_t)a.n_nodes * slices, 1u << 20), kFaceThreads, smem, stream>>>(
        a, slices, cut);
}

template <int kColor>
void launch_colours(const UnitLevelArgs& a, bool any_split, int num_sms, cudaStream_t stream) {
    if (!a.spread) {
        launch_faces<kColor>(a, any_split, num_sms, stream);
        return;
    }
    // about eight blocks per SM, at least one per unit
    uint32_t chunks = 1;
    while (chunks < 64 && (uint64_t)a.n_units * chunks < (uint64_t)std::max(num_sms, 1) * 16) chunks <<= 1;
    k_spread<kColor><<<a.n_units * chunks, kSpreadThreads, 0, stream>>>(a, chunks);
}

}   // namespace

// The colours' kernels, compiled apart: OC_UNITS_PART 0 raw and averaged in the
// cell, 1 inter-cell, 2 distance-weighted.
int launch_units_raw(const UnitLevelArgs& a, bool random, uint32_t mean_candidates, bool any_split, int num_sms,
                     cudaStream_t stream);
int launch_units_intra(const UnitLevelArgs& a, bool random, uint32_t mean_candidates, bool any_split, int num_sms,
                       cudaStream_t stream);
int launch_units_inter(const UnitLevelArgs& a, bool random, uint32_t mean_candidates, bool any_split, int num_sms,
                       cudaStream_t stream);
int launch_units_weighted(const UnitLevelArgs& a, bool random, uint32_t mean_candidates, bool any_split, int num_sms,
                          cudaStream_t stream);

#if OC_UNITS_PART == 1
int launch_units_inter(const UnitLevelArgs& a, bool random, uint32_t mean_candidates, bool any_split, int num_sms,
                       cudaStream_t stream) {
    const int launches = launch_units_as<2>(a, random, mean_candidates, any_split, num_sms, stream);
    launch_colours<2>(a, any_split, num_sms, stream);
    return launches + 1;
}
#elif OC_UNITS_PART == 2
int launch_units_weighted(const UnitLevelArgs& a, bool random, uint32_t mean_candidates, bool any_split, int num_sms,
                          cudaStream_t stream) {
    const int launches = launch_units_as<3>(a, random, mean_candidates, any_split, num_sms, stream);
    launch_colours<3>(a, any_split, num_sms, stream);
    return launches + 1;
}
#else
int launch_units_raw(const UnitLevelArgs& a, bool random, uint32_t mean_candidates, bool any_split, int num_sms,
                     cudaStream_t stream) {
    return launch_units_as<0>(a, random, mean_candidates, any_split, num_sms, stream);
}

int launch_units_intra(const UnitLevelArgs& a, bool random, uint32_t mean_candidates, bool any_split, int num_sms,
                       cudaStream_t stream) {
    return launch_units_as<1>(a, random, mean_candidates, any_split, num_sms, stream);
}

int launch_units_level(const UnitLevelArgs& a, uint32_t mode, uint32_t mean_candidates, bool any_split, int num_sms,
                       cudaStream_t stream) {
    if (!a.n_units) return 0;
    const auto go = (mode & kModeIntra)                                ? launch_units_intra
                    : (mode & kModeInter) && (mode & kModeWeight) ? launch_units_weighted
                    : (mode & kModeInter)                              ? launch_units_inter
                                                                       : launch_units_raw;
    return go(a, (mode & kModeRandom) != 0, mean_candidates, any_split, num_sms, stream);
}

int launch_foreign(const UnitLevelArgs& a, bool colour, int num_sms, cudaStream_t stream) {
    if (!a.n_units) return 0;
    // up to eight blocks per SM; units of a level of few are shared by up to 16
    const uint64_t blocks = (uint64_t)std::max(num_sms, 1) * 8;
    uint32_t chunks = 1;
    while (chunks < 16 && (uint64_t)a.n_units * chunks < blocks) chunks <<= 1;
    k_foreign<<<(unsigned)std::min<uint64_t>((uint64_t)a.n_units * chunks, blocks), kForeignThreads, 0, stream>>>(a, chunks,
                                                                                                          colour);
    return 1;
}

int launch_place_units(const uint64_t* src_off, const uint64_t* dst_off, const uint32_t* count, uint32_t n_nodes,
                       uint64_t n, const uint64_t* total, const OutParams& out, const FixedGrid& fixed,
                       const uint8_t* cloud, uint32_t stride,
                       bool float_input, bool averaged, const uint32_t* stage_lut, const uint64_t* stage_col,
                       uint8_t* rec, uint32_t* err, int num_sms, cudaStream_t stream) {
    if (!n_nodes) return 0;
    auto go = [&](auto kern) {
        // one wave of blocks; fewer for a small cloud
        const uint64_t fit = (uint64_t)std::max(num_sms, 1) *
                             blocks_per_sm(reinterpret_cast<const void*>(kern), 256, 0);
        const unsigned grid = (unsigned)std::max<uint64_t>(1, std::min<uint64_t>(fit, (n + 1023) / 1024));
        kern<<<grid, 256, 0, stream>>>(src_off, dst_off, count, n_nodes, n, total, out, fixed, cloud, stride, stage_lut,
                                       stage_col, rec, err);
    };
    if (float_input) averaged ? go(k_place_units<true, true>) : go(k_place_units<true, false>);
    else averaged ? go(k_place_units<false, true>) : go(k_place_units<false, false>);
    return 1;
}

#endif   // OC_UNITS_PART

}   // namespace oc
