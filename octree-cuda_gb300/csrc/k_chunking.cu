// Chunking stages of the LOD build: binning into the finest counting grid,
// the count pyramid, tree enumeration, leaf tagging and point distribution.
//
// Replaces the reference kernels K1-K5 (point_counting.cuh:29-53,
// point_count_propagation.cuh:34-86, octree_initialization.cuh:24-52,
// hierarchical_merging.cuh:35-122, point_distributing.cuh:30-75).  The dense
// counting grid is kept in Morton order so that the eight children of a cell
// are adjacent: the pyramid is a streaming reduction, and the tree is
// enumerated top-down from the internal nodes only (no dense sweeps over the
// upper levels).
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cstdint>
#include <map>
#include <mutex>
#include <type_traits>
#include <utility>

#include "device_common.cuh"
#include "kernels.h"

namespace oc {

namespace {

constexpr uint32_t kLeafTag = 0x80000000u;
constexpr uint32_t kNoKey = 0xFFFFFFFFu;   // run key of lanes without a point

// Sample of the cloud's order in the words after the error word: runs and
// points (order_sample).
constexpr uint32_t kOrderWord = 4;
constexpr uint32_t kOrderWarps = 64;

__device__ __forceinline__ void set_error(uint32_t* err, uint32_t bit) {
    atomicOr(err, bit);
}

// ---------------------------------------------------------------------------
// Tile pipeline of the two streaming passes over the cloud (counting and
// distribution).  Each block walks tiles blockIdx.x, +gridDim.x, ... of
// `tile` records; tile j+1 is bulk-copied (TMA) into the other of two
// shared-memory buffers while tile j is processed.

// counting: 1024-record tiles, 512 threads
constexpr uint32_t kCountTile = 1024;
constexpr uint32_t kCountThreads = 512;
// Distribution stores each record from its own lane where a leaf's points
// follow each other in the cloud, and brings a leaf's records of a tile
// together in shared memory first where they do not (25.8M-point planes, whose
// points jump between leaves: 1.39 -> 0.88 ms; grouping everything costs the
// 119.7M-point terrain 2.38 -> 3.4 ms).
//   kDirect     896-record tiles, 448 threads (three blocks fit one SM's registers)
//   kGrouped    768-record tiles, one record per thread
//   kByTile     as kDirect; a round of 448 records is grouped when the runs of
//               the tile before were short (float records: with 27-byte tiles
//               its shared memory would take the L1 cache the leaf tags live
//               in, 2.38 -> 2.76 ms)
// A sample of the cloud's order (order_sample) chooses kGrouped or the
// other kernel of the record type.
enum DistMode : int { kDirect, kGrouped, kByTile };
__host__ __device__ constexpr uint32_t dist_threads(int mode) { return mode == kGrouped ? 768 : 448; }
__host__ __device__ constexpr uint32_t dist_tile(int mode) { return mode == kGrouped ? 768 : 896; }
constexpr uint32_t kGroupRun = 4;   // runs of equal leaves shorter than this on average: grouped
constexpr uint64_t kGroupMinPoints = 1 << 18;
constexpr uint32_t kGroupMaxStride = 64;

// Grouping of a round of records (one per thread) by leaf: a hash of the
// leaves, the byte image of the records in leaf order, and per record in that
// order its position and word.
template <int kMode>
struct GroupSmem {
    static constexpr uint32_t kRecords = dist_threads(kMode);
    static constexpr uint32_t kSlots = kMode == kGrouped ? 1024 : 512;
    static constexpr uint32_t kHashShift = kMode == kGrouped ? 22 : 23;
    static constexpr uint32_t kImage = kMode == kGrouped ? 20 * 1024 : 11 * 1024;
    uint32_t key[kSlots];       // leaf + 1, 0 = empty
    uint32_t count[kSlots];     // records
    uint32_t first[kSlots];     // their first position
    uint32_t at[kSlots];        // ... in the image (bytes) << 16 | in leaf order
    uint8_t level[kSlots];      // the leaf's level
    uint32_t pos[kRecords];     // in leaf order
    uint32_t word[kRecords];
    uint16_t rec[kRecords];
    uint16_t runs[kRecords];    // slots in use
    uint32_t warp[32];
    uint32_t n_runs, bytes, bad;   // bytes: of the whole image
    uint32_t lead[3];           // runs of the tile (by tile), the one before, the one after
    uint32_t pad[2];
    uint8_t image[kImage];      // 16-byte aligned
};

__host__ __device__ inline uint32_t align_up(uint32_t x, uint32_t a) {
    return (x + a - 1) / a * a;
}

// Shared-memory layout: [0, 16) two mbarriers, [16, 20) abort flag, then the
// boundary keys of the three axes, the Morton spread table and two tile
// buffers.  A buffer holds a tile's byte span rounded out to 16 bytes plus
// read slack.
struct ChunkSmem {
    uint32_t keys_off, spread_off, buf_off, buf_bytes, total;
};

__host__ __device__ inline ChunkSmem chunk_smem(uint32_t stride, uint32_t grid, bool f32, uint32_t tile,
                                                bool keys = true) {
    ChunkSmem m;
    m.keys_off = 128;
    m.spread_off = align_up(m.keys_off + (keys ? 3 * (grid + 2) * (f32 ? 4u : 8u) : 0u), 16);
    m.buf_off = align_up(m.spread_off + grid * 4, 128);
    m.buf_bytes = align_up(tile * stride + 48, 128);
    m.total = m.buf_off + 2 * m.buf_bytes;
    return m;
}

// Copies the boundary keys and the spread table into shared memory.
template <bool kF32>
__device__ __forceinline__ void load_tables(const CloudGrid& g, uint8_t* smem, const ChunkSmem& L, bool keys = true) {
    using K = typename std::conditional<kF32, int32_t, long long>::type;
    const K* src = static_cast<const K*>(g.keys);
    K* dst = reinterpret_cast<K*>(smem + L.keys_off);
    if (keys)
        for (uint32_t i = threadIdx.x; i < 3 * (g.grid + 2); i += blockDim.x) dst[i] = src[i];
    uint32_t* sp = reinterpret_cast<uint32_t*>(smem + L.spread_off);
    for (uint32_t i = threadIdx.x; i < g.grid; i += blockDim.x) sp[i] = g.spread[i];
}

__device__ __forceinline__ void issue_tile(const uint8_t* __restrict__ cloud, uint64_t n, uint32_t stride, uint32_t tile,
                                           uint64_t t, uint8_t* buf, uint64_t* bar) {
    const uint64_t p0 = t * tile;
    const uint64_t p1 = (n - p0) < tile ? n : p0 + tile;
    const uint64_t a0 = (p0 * stride) & ~15ull, a1 = (p1 * stride + 15) & ~15ull;
    bulk_load(buf, cloud + a0, (uint32_t)(a1 - a0), bar);
}

// Runs body(records_of_tile, first_point, count) for every tile of this
// block.  The body must be memory-safe for any buffer contents: after a
// bounded wait gives up (error bit kErrTimeout) the tile is still processed
// by every thread, so that warp collectives stay converged, and the loop
// ends at the next block barrier.
template <uint32_t kTile, class Body>
__device__ __forceinline__ void tile_loop(const uint8_t* __restrict__ cloud, uint64_t n, uint32_t stride, uint8_t* smem,
                                          const ChunkSmem& L, uint32_t* err, Body&& body) {
    uint64_t* bar = reinterpret_cast<uint64_t*>(smem);
    volatile uint32_t* abort_flag = reinterpret_cast<volatile uint32_t*>(smem + 16);
    uint8_t* buf0 = smem + L.buf_off;
    uint8_t* buf1 = buf0 + L.buf_bytes;
    const uint64_t tiles = (n + kTile - 1) / kTile;
    if (threadIdx.x == 0) {
        mbar_init(&bar[0], 1);
        mbar_init(&bar[1], 1);
        *abort_flag = 0;
        fence_barrier_init();
    }
    __syncthreads();
    uint64_t t = blockIdx.x;
    if (threadIdx.x == 0 && t < tiles) issue_tile(cloud, n, stride, kTile, t, buf0, &bar[0]);
    uint32_t j = 0;
    bool aborted = false;
    for (; t < tiles; t += gridDim.x, ++j) {
        const uint32_t slot = j & 1;
        const uint64_t tn = t + gridDim.x;
        // the other buffer was released by the barrier that ended the previous tile
        if (threadIdx.x == 0 && tn < tiles) issue_tile(cloud, n, stride, kTile, tn, slot ? buf0 : buf1, &bar[slot ^ 1]);
        if (!mbar_wait_bounded(&bar[slot], (j >> 1) & 1)) {
            set_error(err, kErrTimeout);
            *abort_flag = 1;
        }
        const uint64_t p0 = t * kTile;
        const uint32_t cnt = (uint32_t)((n - p0) < kTile ? (n - p0) : kTile);
        body((slot ? buf1 : buf0) + (uint32_t)((p0 * stride) & 15), p0, cnt);
        __syncthreads();
        if (*abort_flag) {
            aborted = true;
            break;
        }
    }
    if (aborted && threadIdx.x == 0) {
        // let the copies still in flight land before the block exits (bounded)
        const uint32_t slot = j & 1;
        mbar_wait_bounded(&bar[slot], (j >> 1) & 1);
        if (t + gridDim.x < tiles) mbar_wait_bounded(&bar[slot ^ 1], ((j + 1) >> 1) & 1);
    }
}

// Cells of a point from its coordinate words (3 floats or 3 x lo/hi of
// doubles), exactly as (int64)fmin((p - min) / t, G - 1) in binary64.
// Returns false when the point lies below the bounding box.
template <bool kF32>
__device__ __forceinline__ bool point_cells(const uint32_t* w, const CloudGrid& g, const uint8_t* smem,
                                            const ChunkSmem& L, int cell[3]) {
    const uint32_t G = g.grid;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        int i;
        if (kF32) {
            const int32_t* K = reinterpret_cast<const int32_t*>(smem + L.keys_off) + a * (G + 2);
            const uint32_t b = w[a];
            i = table_cell<int32_t>(dev_key32(b), __fmaf_rn(__uint_as_float(b), g.r[a], g.c[a]), K, G);
            if (i == -2) i = exact_axis_cell((double)__uint_as_float(b), g.ax[a].mn, g.ax[a].t, G);
        } else {
            const long long* K = reinterpret_cast<const long long*>(smem + L.keys_off) + a * (G + 2);
            const uint32_t lo = w[2 * a], hi = w[2 * a + 1];
            i = table_cell<long long>(dev_key64(lo, hi), __fmaf_rn(approx_f64(lo, hi), g.r[a], g.c[a]), K, G);
            if (i == -2) i = exact_axis_cell(__hiloint2double((int)hi, (int)lo), g.ax[a].mn, g.ax[a].t, G);
        }
        cell[a] = i;
    }
    return (cell[0] | cell[1] | cell[2]) >= 0;
}

__device__ __forceinline__ uint32_t cell_morton(const int cell[3], const uint8_t* smem, const ChunkSmem& L) {
    const uint32_t* sp = reinterpret_cast<const uint32_t*>(smem + L.spread_off);
    return (sp[cell[0]] << 2) | (sp[cell[1]] << 1) | sp[cell[2]];
}

// K1 (point_counting.cuh:29-53): points per finest cell.  Consecutive lanes
// in the same cell add their count with one atomic.
// With `occ` (sparse clouds) the run leaders also flag their cell's 64-cell
// block (a level-2 cell): a plain byte store, no read-modify-write.
template <bool kF32>
__global__ void __launch_bounds__(kCountThreads) k_count(const uint8_t* __restrict__ cloud, uint64_t n, uint32_t stride,
                                                         CloudGrid g, uint32_t* __restrict__ pyr0, uint8_t* occ,
                                                         uint32_t* err) {
    extern __shared__ __align__(128) uint8_t smem[];
    const ChunkSmem L = chunk_smem(stride, g.grid, kF32, kCountTile);
    load_tables<kF32>(g, smem, L);
    const uint32_t lane = threadIdx.x & 31;
    tile_loop<kCountTile>(cloud, n, stride, smem, L, err, [&](const uint8_t* recs, uint64_t p0, uint32_t cnt) {
#pragma unroll 1
        for (uint32_t base = 0; base < kCountTile; base += kCountThreads) {
            const uint32_t k = base + threadIdx.x;
            uint32_t m = kNoKey;
            if (k < cnt) {
                constexpr int kWords = kF32 ? 3 : 6;
                uint32_t w[kWords];
                record_words<kWords>(recs + (uint64_t)k * stride, w);
                int cell[3];
                if (point_cells<kF32>(w, g, smem, L, cell)) m = cell_morton(cell, smem, L);
                else set_error(err, kErrBelowBox);
            }
            const uint32_t starts = run_starts(m);
            if (m != kNoKey && ((starts >> lane) & 1u)) {
                atomicAdd(&pyr0[m], run_end(starts) - lane);
                if (occ) occ[m >> 6] = 1;
            }
        }
    });
}

// Coordinate minima and maxima (calculateRealBB, src/boundingbox.h:11-33) as
// ordered keys: keys[0..2] minima, keys[3..5] maxima.  NaN coordinates are
// skipped, as fmin / fmax skip them.  Float keys are widened to 64 bits.
template <bool kF32>
__global__ void __launch_bounds__(256) k_bbox(const uint8_t* __restrict__ cloud, uint64_t n, uint32_t stride,
                                              long long* keys) {
    long long mn[3] = {LLONG_MAX, LLONG_MAX, LLONG_MAX}, mx[3] = {LLONG_MIN, LLONG_MIN, LLONG_MIN};
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        constexpr int kWords = kF32 ? 3 : 6;
        uint32_t w[kWords];
        const uint8_t* rec = cloud + i * stride;
        const uintptr_t a = reinterpret_cast<uintptr_t>(rec);
        const uint32_t* q = reinterpret_cast<const uint32_t*>(a & ~(uintptr_t)3);
        const uint32_t sh = (uint32_t)(a & 3) * 8;
#pragma unroll
        for (int j = 0; j < kWords; ++j) w[j] = __funnelshift_r(q[j], q[j + 1], sh);
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            long long k;
            bool nan;
            if (kF32) {
                nan = (w[c] & 0x7FFFFFFFu) > 0x7F800000u;
                k = dev_key32(w[c]);
            } else {
                const uint32_t lo = w[2 * c], hi = w[2 * c + 1];
                nan = (hi & 0x7FFFFFFFu) > 0x7FF00000u || ((hi & 0x7FFFFFFFu) == 0x7FF00000u && lo != 0);
                k = dev_key64(lo, hi);
            }
            if (!nan) {
                mn[c] = min(mn[c], k);
                mx[c] = max(mx[c], k);
            }
        }
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        for (int o = 16; o > 0; o >>= 1) {
            mn[c] = min(mn[c], (long long)__shfl_xor_sync(0xffffffffu, (unsigned long long)mn[c], o));
            mx[c] = max(mx[c], (long long)__shfl_xor_sync(0xffffffffu, (unsigned long long)mx[c], o));
        }
    }
    if ((threadIdx.x & 31) == 0) {
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            if (mn[c] != LLONG_MAX) atomicMin(&keys[c], mn[c]);
            if (mx[c] != LLONG_MIN) atomicMax(&keys[3 + c], mx[c]);
        }
    }
}

__global__ void k_bbox_init(long long* keys) {
    if (threadIdx.x < 6) keys[threadIdx.x] = threadIdx.x < 3 ? LLONG_MAX : LLONG_MIN;
}

// Level l -> levels l+1 and l+2.  A warp reads 16 level-(l+2) cells' 64
// Morton-contiguous counts each, 512 bytes per load and eight loads in flight
// (bound by DRAM; a thread per level-(l+2) cell, whose loads lie 256 bytes
// apart, reached 4.9 TB/s; 134M cells and the
// upper levels 150 -> 112 us).
constexpr uint32_t kPyramidCells = 8 * 16;   // per block of 256

__global__ void __launch_bounds__(256) k_pyramid2(const uint32_t* __restrict__ src, uint32_t* __restrict__ dst1,
                                                  uint32_t* __restrict__ dst2, uint64_t n2, uint32_t* nz_src,
                                                  uint32_t* nz_dst1) {
    __shared__ uint32_t s_nz[2];
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint64_t first = blockIdx.x * (uint64_t)kPyramidCells + warp * 16;
    if (threadIdx.x < 2) s_nz[threadIdx.x] = 0;
    __syncthreads();
    uint4 v[8];
#pragma unroll
    for (uint32_t j = 0; j < 8; ++j) {
        const uint64_t cell = first + 2 * j + (lane >> 4);
        v[j] = cell < n2 ? reinterpret_cast<const uint4*>(src)[cell * 16 + (lane & 15)] : make_uint4(0, 0, 0, 0);
    }
    uint32_t nzs = 0, nzd = 0;
#pragma unroll
    for (uint32_t j = 0; j < 8; ++j) {
        const uint64_t cell = first + 2 * j + (lane >> 4);
        nzs += (v[j].x != 0) + (v[j].y != 0) + (v[j].z != 0) + (v[j].w != 0);
        uint32_t sum = v[j].x + v[j].y + v[j].z + v[j].w;
        sum += __shfl_xor_sync(0xffffffffu, sum, 1);
        if (cell < n2 && !(lane & 1)) {
            dst1[cell * 8 + ((lane & 15) >> 1)] = sum;
            nzd += sum != 0;
        }
        sum += __shfl_xor_sync(0xffffffffu, sum, 2);
        sum += __shfl_xor_sync(0xffffffffu, sum, 4);
        sum += __shfl_xor_sync(0xffffffffu, sum, 8);
        if (cell < n2 && !(lane & 15)) dst2[cell] = sum;
    }
    nzs = __reduce_add_sync(0xffffffffu, nzs);
    nzd = __reduce_add_sync(0xffffffffu, nzd);
    if (lane == 0) {
        if (nzs) atomicAdd(&s_nz[0], nzs);
        if (nzd) atomicAdd(&s_nz[1], nzd);
    }
    __syncthreads();
    if (threadIdx.x == 0 && s_nz[0]) atomicAdd(nz_src, s_nz[0]);
    if (threadIdx.x == 1 && s_nz[1]) atomicAdd(nz_dst1, s_nz[1]);
}

// The same for the finest level of a sparse cloud: a level-2 cell whose block
// flag is clear has only empty children, and its sums stay the zeros that the
// pyramid of such a cloud starts from (writing them, 75 MB of a grid of 512,
// took 6 of 46 us).  One thread per level-2 cell (with the warps of k_pyramid2
// the level of 134M cells took 72 us, 5M points, instead of 48).
__global__ void k_pyramid2_sparse(const uint32_t* __restrict__ src, uint32_t* __restrict__ dst1, uint32_t* __restrict__ dst2,
                                  uint64_t n2, uint32_t* nz_src, uint32_t* nz_dst1, const uint8_t* __restrict__ occ) {
    uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    uint32_t nzs = 0, nzd = 0;
    if (i < n2 && occ[i]) {
        const uint4* s = reinterpret_cast<const uint4*>(src + i * 64);
        uint32_t sums[8];
        uint32_t total = 0;
#pragma unroll
        for (int c = 0; c < 8; ++c) {
            uint4 a = s[2 * c], b = s[2 * c + 1];
            uint32_t v = a.x + a.y + a.z + a.w + b.x + b.y + b.z + b.w;
            nzs += (a.x != 0) + (a.y != 0) + (a.z != 0) + (a.w != 0) + (b.x != 0) + (b.y != 0) + (b.z != 0) + (b.w != 0);
            sums[c] = v;
            nzd += v != 0;
            total += v;
        }
        uint4* d = reinterpret_cast<uint4*>(dst1 + i * 8);
        d[0] = make_uint4(sums[0], sums[1], sums[2], sums[3]);
        d[1] = make_uint4(sums[4], sums[5], sums[6], sums[7]);
        dst2[i] = total;
    }
    for (int o = 16; o > 0; o >>= 1) {
        nzs += __shfl_down_sync(0xffffffffu, nzs, o);
        nzd += __shfl_down_sync(0xffffffffu, nzd, o);
    }
    if ((threadIdx.x & 31) == 0) {
        if (nzs) atomicAdd(nz_src, nzs);
        if (nzd) atomicAdd(nz_dst1, nzd);
    }
}

// Block-wide exclusive scan of one value per thread (blockDim.x = 1024).
__device__ __forceinline__ uint32_t block_exclusive_scan(uint32_t v, uint32_t* warp_sums, uint32_t& total) {
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= (uint32_t)o) x += y;
    }
    if (lane == 31) warp_sums[warp] = x;
    __syncthreads();
    if (warp == 0) {
        uint32_t w = lane < (blockDim.x >> 5) ? warp_sums[lane] : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            uint32_t y = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= (uint32_t)o) w += y;
        }
        warp_sums[lane] = w;
    }
    __syncthreads();
    uint32_t warp_prefix = warp ? warp_sums[warp - 1] : 0;
    total = warp_sums[(blockDim.x >> 5) - 1];
    __syncthreads();
    return warp_prefix + x - v;
}

// Top-down tree enumeration in hierarchy BFS order (potree_exporter.cu:62-96):
// a node at level >= 1 whose count reaches the threshold is internal
// (hierarchical_merging.cuh:134) and all its occupied children are tree nodes;
// every other tree node is a leaf.  One block walks the levels, after it summed
// up the top of the pyramid, levels of at most kTopCells cells, in shared
// memory: those are bound by launches (a launch per two levels and one for the
// root: pyramid and tree took 32 us on a grid of 128 and 56 of 512, now 21 and
// 46; 2M points 0.475 -> 0.466 ms).
constexpr uint32_t kTopCells = 32768;

// First level of at most kTopCells cells, counted in steps of two.
inline uint32_t top_level(uint32_t depth) {
    uint32_t l = 0;
    while (depth >= l && (1ull << (3 * (depth - l))) > kTopCells) l += 2;
    return l;
}

__global__ void __launch_bounds__(1024) k_enumerate(uint32_t* pyr, const uint64_t* __restrict__ loff, uint32_t depth,
                                                    uint32_t from, uint32_t* nonzero, uint32_t threshold, uint32_t* key,
                                                    uint32_t* count, uint8_t* level, uint16_t* info,
                                                    uint32_t* child_first, uint32_t cap, uint32_t* level_start,
                                                    uint32_t* n_nodes, uint32_t* err) {
    __shared__ uint32_t warp_sums[32];
    __shared__ uint32_t s_next;
    __shared__ __align__(16) uint32_t s_cells[kTopCells / 8];
    __shared__ uint32_t s_nz[32];
    if (threadIdx.x < 32) s_nz[threadIdx.x] = 0;
    __syncthreads();
    for (uint32_t l = from; l < depth; ++l) {
        constexpr uint32_t kPer = kTopCells / 8 / 1024;
        const uint32_t n1 = 1u << (3 * (depth - l - 1));   // cells of level l + 1: at most kTopCells / 8
        const uint4* src = reinterpret_cast<const uint4*>(l == from ? pyr + loff[l] : s_cells);
        uint32_t sum[kPer], nz = 0;
#pragma unroll
        for (uint32_t j = 0; j < kPer; ++j) {
            const uint32_t i = threadIdx.x + j * 1024;
            sum[j] = 0;
            if (i < n1) {
                const uint4 a = src[2 * i], b = src[2 * i + 1];
                sum[j] = a.x + a.y + a.z + a.w + b.x + b.y + b.z + b.w;
                nz += (a.x != 0) + (a.y != 0) + (a.z != 0) + (a.w != 0) + (b.x != 0) + (b.y != 0) + (b.z != 0) +
                      (b.w != 0);
            }
        }
        nz = __reduce_add_sync(0xffffffffu, nz);
        if ((threadIdx.x & 31) == 0 && nz) atomicAdd(&s_nz[l], nz);
        __syncthreads();   // the level below is read
#pragma unroll
        for (uint32_t j = 0; j < kPer; ++j) {
            const uint32_t i = threadIdx.x + j * 1024;
            if (i < n1) pyr[loff[l + 1] + i] = s_cells[i] = sum[j];
        }
        __syncthreads();
    }
    if (threadIdx.x >= from && threadIdx.x < depth) nonzero[threadIdx.x] = s_nz[threadIdx.x];
    if (threadIdx.x == depth) nonzero[depth] = pyr[loff[depth]] != 0;
    if (threadIdx.x == 0) {
        key[0] = 0;
        count[0] = pyr[loff[depth]];
        level[0] = (uint8_t)depth;
        s_next = 1;
        level_start[depth] = 0;
    }
    __syncthreads();
    uint32_t cur_begin = 0, cur_end = 1;
    for (int l = (int)depth; l >= 1; --l) {
        for (uint32_t base = cur_begin; base < cur_end; base += blockDim.x) {
            uint32_t i = base + threadIdx.x;
            uint32_t mask = 0;
            bool internal = false;
            uint32_t k = 0;
            if (i < cur_end) {
                k = key[i];
                internal = count[i] >= threshold;
                if (internal) {
                    const uint4* c = reinterpret_cast<const uint4*>(pyr + loff[l - 1] + (uint64_t)k * 8);
                    uint4 a = c[0], b = c[1];
                    mask = (a.x != 0) | ((a.y != 0) << 1) | ((a.z != 0) << 2) | ((a.w != 0) << 3) | ((b.x != 0) << 4) |
                           ((b.y != 0) << 5) | ((b.z != 0) << 6) | ((b.w != 0) << 7);
                }
            }
            uint32_t total;
            uint32_t off = block_exclusive_scan(__popc(mask), warp_sums, total);
            uint32_t next = s_next;
            if (i < cur_end) {
                info[i] = (uint16_t)((internal ? 1u : 0u) | (mask << 1));
                child_first[i] = internal ? next + off : 0xFFFFFFFFu;
                if (internal) {
                    const uint32_t* c = pyr + loff[l - 1] + (uint64_t)k * 8;
                    uint32_t j = next + off;
                    for (uint32_t s = 0; s < 8; ++s) {
                        if (!(mask & (1u << s))) continue;
                        if (j < cap) {
                            key[j] = k * 8 + s;
                            count[j] = c[s];
                            level[j] = (uint8_t)(l - 1);
                        }
                        ++j;
                    }
                }
            }
            __syncthreads();
            if (threadIdx.x == 0) {
                s_next = next + total;
                if (s_next > cap) set_error(err, kErrNodeCap);
            }
            __syncthreads();
            if (s_next > cap) return;
        }
        cur_begin = cur_end;
        cur_end = s_next;
        if (threadIdx.x == 0) level_start[l - 1] = cur_begin;
    }
    // level-0 nodes are leaves
    for (uint32_t i = cur_begin + threadIdx.x; i < cur_end; i += blockDim.x) {
        info[i] = 0;
        child_first[i] = 0xFFFFFFFFu;
    }
    if (threadIdx.x == 0) {
        *n_nodes = cur_end;
        level_start[depth + 1] = cur_end;
    }
}

// Leaf data offsets and leaf tags from the node table, without the host: one
// block scans the nodes in BFS order.  Leaf i gets data_idx = the points of
// the leaves before it (hierarchy BFS order), its pyramid cell the tag
// kLeafTag | i, and its fill counter 0.  Skipped when the node table
// overflowed; flags kErrTag when the leaves do not hold all n_points.
__global__ void __launch_bounds__(1024) k_leaf_prep(const uint32_t* __restrict__ n_nodes_p,
                                                    const uint16_t* __restrict__ info, const uint32_t* __restrict__ count,
                                                    const uint8_t* __restrict__ level, const uint32_t* __restrict__ key,
                                                    uint32_t* pyr, const uint64_t* __restrict__ loff, uint64_t* data_idx,
                                                    uint32_t* fill, uint64_t n_points, uint32_t* err) {
    __shared__ uint64_t warp_sums[32];
    if (*err & kErrNodeCap) return;
    const uint32_t n = *n_nodes_p;
    uint64_t running = 0;
    for (uint32_t k0 = 0; k0 < n; k0 += blockDim.x) {
        const uint32_t i = k0 + threadIdx.x;
        const bool leaf = i < n && !(info[i] & 1);
        const uint64_t c = leaf ? count[i] : 0;
        uint64_t tot;
        const uint64_t pre = block_exclusive_scan64(c, warp_sums, tot);
        if (i < n) {
            fill[i] = 0;
            data_idx[i] = leaf ? (running + pre) | ((uint64_t)level[i] << kLeafLevelShift) : 0;
            if (leaf) pyr[loff[level[i]] + key[i]] = kLeafTag | i;
        }
        running += tot;
    }
    if (threadIdx.x == 0 && running != n_points) set_error(err, kErrTag);
}

// How far the cloud's order keeps leaves together: runs of points in one block
// of 16^3 finest cells, about a leaf's size, among 32 consecutive points at
// kOrderWarps places of the cloud.  Approximate cells do.
template <bool kF32>
__device__ __forceinline__ void order_sample(const uint8_t* __restrict__ cloud, uint64_t n, uint32_t stride,
                                             const CloudGrid& g, uint32_t sample, uint32_t* order) {
    const uint32_t lane = threadIdx.x & 31;
    if (n < 32 || sample >= kOrderWarps) return;
    const uint64_t p = (n - 32) * sample / (kOrderWarps - 1) + lane;
    constexpr int kWords = kF32 ? 3 : 6;
    uint32_t w[kWords], block = 0;
    record_words<kWords>(cloud + p * stride, w);
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const float v = kF32 ? __uint_as_float(w[a]) : approx_f64(w[kF32 ? 0 : 2 * a], w[kF32 ? 0 : 2 * a + 1]);
        const float u = fminf(fmaxf(__fmaf_rn(v, g.r[a], g.c[a]), 0.0f), (float)(g.grid - 1));
        block = (block << 10) | ((uint32_t)u >> 4);
    }
    const uint32_t runs = __popc(run_starts(block));
    if (lane == 0) {
        atomicAdd(order, runs);
        atomicAdd(order + 1, 32u);
    }
}

// Writes the leaf tag of every occupied finest cell into the cell: one
// thread per level-1 cell reads its 8 children and, when some of them are
// occupied and untagged, the nearest tagged ancestor.
__global__ void k_push_tags(uint32_t* __restrict__ pyr, const uint64_t* __restrict__ loff, uint32_t depth, uint64_t n1,
                            const uint8_t* __restrict__ occ, uint32_t* err, const uint8_t* __restrict__ cloud,
                            uint64_t n, uint32_t stride, uint32_t float_input, CloudGrid g, uint32_t tag_blocks) {
    if (blockIdx.x >= tag_blocks) {   // the blocks after those of the tags sample the cloud's order
        const uint32_t sample = (blockIdx.x - tag_blocks) * (blockDim.x / 32) + threadIdx.x / 32;
        if (float_input) order_sample<true>(cloud, n, stride, g, sample, err + kOrderWord);
        else order_sample<false>(cloud, n, stride, g, sample, err + kOrderWord);
        return;
    }
    const uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    if (i >= n1) return;
    if (occ && occ[i >> 3] == 0) return;   // no point in this 64-cell block
    if (pyr[loff[1] + i] == 0) return;     // none in these 8 cells: an eighth of the bytes, where most are empty
    uint4* c = reinterpret_cast<uint4*>(pyr + i * 8);
    uint4 a = c[0], b = c[1];
    uint32_t v[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
    bool need = false;
#pragma unroll
    for (int s = 0; s < 8; ++s) need |= v[s] != 0 && !(v[s] & kLeafTag);
    if (!need) return;
    uint32_t tag = 0;
    uint64_t k = i;
    for (uint32_t l = 1; l <= depth; ++l, k >>= 3) {
        const uint32_t w = pyr[loff[l] + k];
        if (w & kLeafTag) {
            tag = w;
            break;
        }
    }
    if (!tag) {
        set_error(err, kErrTag);
        return;
    }
#pragma unroll
    for (int s = 0; s < 8; ++s)
        if (v[s] != 0 && !(v[s] & kLeafTag)) v[s] = tag;
    c[0] = make_uint4(v[0], v[1], v[2], v[3]);
    c[1] = make_uint4(v[4], v[5], v[6], v[7]);
}

// Reserves every leaf's records of the round with one atomic and lays out the
// image: a leaf's part starts at the 16-byte phase of its destination.  All
// threads; starts after a barrier, ends with one.
template <int kMode>
__device__ __forceinline__ void group_place(GroupSmem<kMode>& gs, const uint64_t* __restrict__ data_idx, uint32_t* fill,
                                            uint64_t n) {
    constexpr uint32_t kGroupSlots = GroupSmem<kMode>::kSlots;
    static_assert(kGroupSlots <= 2 * dist_threads(kMode), "two slots per thread");
    const uint32_t t = threadIdx.x, lane = t & 31, warp = t >> 5;
    uint32_t c[2] = {0, 0}, v[2] = {0, 0}, f[2];
    if (t < kGroupSlots / 2) {
#pragma unroll
        for (uint32_t j = 0; j < 2; ++j) {
            c[j] = gs.count[2 * t + j];
            f[j] = c[j] ? atomicAdd(&fill[gs.key[2 * t + j] - 1], c[j]) : 0u;
        }
#pragma unroll
        for (uint32_t j = 0; j < 2; ++j) {
            if (!c[j]) continue;
            const uint32_t s = 2 * t + j;
            const uint64_t d = data_idx[gs.key[s] - 1];
            f[j] += (uint32_t)d;
            if ((uint64_t)f[j] + c[j] > n) gs.bad = 1;   // only reachable with corrupted input tags
            gs.first[s] = f[j];
            gs.level[s] = (uint8_t)(d >> kLeafLevelShift);
            v[j] = ((((f[j] * 18u) & 15u) + c[j] * 18u + 15u) & ~15u) << 16 | c[j];
            gs.runs[atomicAdd(&gs.n_runs, 1u)] = (uint16_t)s;
        }
    }
    const uint32_t sum = v[0] + v[1];
    uint32_t incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= (uint32_t)o) incl += y;
    }
    if (lane == 31) gs.warp[warp] = incl;
    __syncthreads();
    uint32_t run = incl - sum;
    for (uint32_t q = 0; q < kGroupSlots / 64; ++q) run += q < warp ? gs.warp[q] : 0u;
    if (t < kGroupSlots / 2) {
        gs.at[2 * t] = run + (((f[0] * 18u) & 15u) << 16);
        gs.at[2 * t + 1] = run + v[0] + (((f[1] * 18u) & 15u) << 16);
        if (t == kGroupSlots / 2 - 1) gs.bytes = (run + sum) >> 16;
    }
    __syncthreads();
}

// Copies the image out, a warp per leaf: 16-byte words, and 2-byte words at
// both ends; then indices and words, neighbouring lanes to neighbouring
// positions.
template <int kMode>
__device__ __forceinline__ void group_store(const GroupSmem<kMode>& gs, uint64_t p0, uint32_t* __restrict__ lut,
                                            uint32_t* __restrict__ word, uint8_t* __restrict__ rec) {
    constexpr uint32_t kGroupSlots = GroupSmem<kMode>::kSlots;
    const uint32_t t = threadIdx.x, lane = t & 31;
    for (uint32_t r = t >> 5; r < gs.n_runs; r += dist_threads(kMode) / 32) {
        const uint32_t s = gs.runs[r], a0 = gs.at[s] >> 16, a1 = a0 + gs.count[s] * 18u;
        uint8_t* out = rec + (uint64_t)gs.first[s] * 18 - a0;   // of image byte 0
        const uint32_t b0 = (a0 + 15u) & ~15u, b1 = a1 & ~15u;
        if (b0 < b1) {
            for (uint32_t i = b0 + 16 * lane; i < b1; i += 512)
                *reinterpret_cast<uint4*>(out + i) = *reinterpret_cast<const uint4*>(gs.image + i);
            // up to seven 2-byte words before, up to seven after
            const uint32_t i = lane < 8 ? a0 + 2 * lane : b1 + 2 * (lane - 8);
            if (lane < 16 && i < (lane < 8 ? b0 : a1))
                *reinterpret_cast<uint16_t*>(out + i) = *reinterpret_cast<const uint16_t*>(gs.image + i);
        } else {
            const uint32_t i = a0 + 2 * lane;   // at most 30 bytes
            if (i < a1) *reinterpret_cast<uint16_t*>(out + i) = *reinterpret_cast<const uint16_t*>(gs.image + i);
        }
    }
    const uint32_t last = gs.at[kGroupSlots - 1], total = (last & 0xFFFFu) + gs.count[kGroupSlots - 1];
    if (t < total) {
        const uint32_t pos = gs.pos[t];
        lut[pos] = (uint32_t)(p0 + gs.rec[t]);
        word[pos] = gs.word[t];
    }
}

template <int kMode>
__device__ __forceinline__ void group_clear(GroupSmem<kMode>& gs) {
    for (uint32_t i = threadIdx.x; i < GroupSmem<kMode>::kSlots; i += dist_threads(kMode)) gs.key[i] = gs.count[i] = 0;
    if (threadIdx.x == 0) gs.n_runs = gs.bad = 0;
}

// K5 (point_distributing.cuh:30-75): every point goes to its leaf's bucket
// with its LUT entry and 18-byte output record.  The first lane of each run
// of equal cells reads the cell's leaf tag; the first lane of each run of
// equal leaves reserves the run's slots with one atomic.  At most 40
// registers, so that three 448-thread blocks share an SM (47 registers leave
// room for two: 119.7M-point build 2.73 -> 2.56 ms).
// kCells: the cell words of octant subsampling instead of sub-step words.  The
// finest cell gives the counting cell as well (its upper bits), so the
// boundary-key lookup is left out; a point beside a boundary of the counting
// grid is evaluated in binary64.
// Positions are in fixed point: the kernel is bound by the issue of
// instructions (70% of the slots), and with float-float positions a third of
// its 490 per point were these (119.7M binary64 points 2.42 -> 2.05 ms, 12.3M
// 0.263 -> 0.229 ms).  Counting, which waits for its atomics, gains nothing by
// them and keeps the boundary keys (0.90 ms either way).
template <bool kF32, bool kCells, int kMode>
__global__ void __launch_bounds__(dist_threads(kMode), kMode == kGrouped ? 2 : 3)
    k_distribute(const uint8_t* __restrict__ cloud, uint64_t n,
                                                              uint32_t stride, CloudGrid g,
                                                              const __grid_constant__ OutParams op,
                                                              const __grid_constant__ FixedGrid fg,
                                                              const uint32_t* __restrict__ pyr0,
                                                              const uint64_t* __restrict__ data_idx, uint32_t* fill,
                                                              uint32_t* __restrict__ lut, uint8_t* __restrict__ rec,
                                                              uint32_t* __restrict__ frac, uint32_t* err,
                                                              const uint32_t* __restrict__ order) {
    extern __shared__ __align__(128) uint8_t smem[];
    // of the two kernels launched, the one for the order of the points runs
    if (order && (order[0] * kGroupRun > order[1]) != (kMode == kGrouped)) return;
    constexpr uint32_t kTile = dist_tile(kMode), kThreads = dist_threads(kMode);
    const ChunkSmem L = chunk_smem(stride, g.grid, kF32, kTile, !kCells);
    load_tables<kF32>(g, smem, L, !kCells);
    GroupSmem<kMode>* gs = reinterpret_cast<GroupSmem<kMode>*>(smem + align_up(L.total, 16));
    if (kMode != kDirect) {   // (tile_loop starts with a barrier)
        group_clear(*gs);
        if (threadIdx.x < 3) gs->lead[threadIdx.x] = 0;
    }
    uint32_t next_turn = 0;
    const uint32_t lane = threadIdx.x & 31;
    tile_loop<kTile>(cloud, n, stride, smem, L, err, [&](const uint8_t* recs, uint64_t p0, uint32_t cnt) {
        bool group = kMode == kGrouped;
        const uint32_t turn = next_turn;
        if (kMode == kByTile) {
            next_turn = turn == 2 ? 0 : turn + 1;
            group = gs->lead[turn == 0 ? 2 : turn - 1] * kGroupRun > kTile;
            if (threadIdx.x == 0) gs->lead[next_turn] = 0;
        }
#pragma unroll 1
        for (uint32_t base = 0; base < kTile; base += kThreads) {
            const uint32_t k = base + threadIdx.x;
            constexpr int kWords = kF32 ? 4 : 7;
            uint32_t w[kWords];
            uint32_t m = kNoKey;
            int32_t q[3];      // kCells: output coordinates, finest cells, colour
            uint32_t fine[3];
            bool proven = true, known[3];   // cells; output coordinates
            uint32_t edge = 0;              // boundary_cells
            if (k < cnt) {
                record_words<kWords>(recs + (uint64_t)k * stride, w);
                int cell[3];
                if (kCells) {
#pragma unroll
                    for (int a = 0; a < 3; ++a) {
                        uint64_t d;
                        bool exact_cell;
                        const bool in = fixed_difference(word_coord<kF32>(w, a), fg.ax[a].o, d);
                        fine[a] = fixed_units(d, fg.ax[a].cell, exact_cell);
                        q[a] = (int32_t)fixed_units(d, fg.ax[a].out, known[a]);
                        cell[a] = (int)(fine[a] >> 6);
                        proven &= in && exact_cell && fine[a] < fg.cells;
                        known[a] = known[a] && in && q[a] >= 0;
                    }
                    if (!(known[0] && known[1] && known[2])) {
#pragma unroll
                        for (int a = 0; a < 3; ++a)
                            if (!known[a]) q[a] = formula_out_coord<kF32>(w, a, op.ax[a]);
                    }
                    if (!proven) {
                        const uint4 c = boundary_cells<kF32>(recs + (uint64_t)k * stride, fg);
                        fine[0] = c.x;
                        fine[1] = c.y;
                        fine[2] = c.z;
                        edge = c.w;
#pragma unroll
                        for (int a = 0; a < 3; ++a)   // (64: a boundary of the counting grid)
                            cell[a] = edge < 64 ? (int)(fine[a] >> 6)
                                                : exact_axis_cell(word_coord_exact<kF32>(w, a), g.ax[a].mn, g.ax[a].t, g.grid);
                    }
                    if ((cell[0] | cell[1] | cell[2]) >= 0) m = cell_morton(cell, smem, L);
                    else set_error(err, kErrBelowBox);
                } else {
                    if (point_cells<kF32>(w, g, smem, L, cell)) m = cell_morton(cell, smem, L);
                    else set_error(err, kErrBelowBox);
                }
            }
            uint32_t starts = run_starts(m);
            uint32_t leader = run_leader(starts);
            uint32_t tag = (m != kNoKey && lane == leader) ? pyr0[m] : 0u;
            tag = __shfl_sync(0xffffffffu, tag, leader);
            uint32_t node = kNoKey;
            if (m != kNoKey) {
                if (tag & kLeafTag) node = tag & ~kLeafTag;
                else set_error(err, kErrTag);
            }
            starts = run_starts(node);
            leader = run_leader(starts);
            const bool lead = node != kNoKey && lane == leader;
            uint64_t first = 0;   // the leaf's level above kLeafLevelShift
            uint32_t slot = 0, rank = lane - leader;
            if (kMode == kByTile) {
                const uint32_t leads = __popc(__ballot_sync(0xffffffffu, lead));
                if (lane == 0) atomicAdd(&gs->lead[turn], leads);
            }
            if (!group) {
                if (lead) first = data_idx[node] + atomicAdd(&fill[node], run_end(starts) - lane);
                first = ((uint64_t)__shfl_sync(0xffffffffu, (uint32_t)(first >> 32), leader) << 32) |
                        __shfl_sync(0xffffffffu, (uint32_t)first, leader);
            } else {
                if (lead) {
                    slot = (node * 2654435761u) >> GroupSmem<kMode>::kHashShift;
                    for (uint32_t probe = 0; probe < GroupSmem<kMode>::kSlots; ++probe) {   // fewer leaves than slots
                        const uint32_t old = atomicCAS(&gs->key[slot], 0u, node + 1);
                        if (old == 0 || old == node + 1) break;
                        slot = (slot + 1) % GroupSmem<kMode>::kSlots;
                    }
                    rank = atomicAdd(&gs->count[slot], run_end(starts) - lane);
                }
                slot = __shfl_sync(0xffffffffu, slot, leader);
                rank = __shfl_sync(0xffffffffu, rank, leader) + lane - leader;
                __syncthreads();
                group_place(*gs, data_idx, fill, n);
                first = gs->first[slot] | ((uint64_t)gs->level[slot] << kLeafLevelShift);
            }
            const uint32_t lv = (uint32_t)(first >> kLeafLevelShift);
            first &= (1ull << kLeafLevelShift) - 1;
            const bool image = group && gs->bytes <= GroupSmem<kMode>::kImage && !gs->bad;
            uint32_t nw[5] = {0, 0, 0, 0, 0};
            bool ok = false;
            const uint64_t pos = first + rank;
            uint32_t fw = 0;
            if (node != kNoKey) {
                if (pos >= n) {   // only reachable with corrupted input tags
                    set_error(err, kErrTag);
                } else {
                    ok = true;
                    const uint32_t col = w[kF32 ? 3 : 6];
                    int32_t x, y, z;
                    if (kCells) {
                        x = q[0];
                        y = q[1];
                        z = q[2];
                        fw = word_edge(edge) | ((fine[0] >> lv) & 127u) | (((fine[1] >> lv) & 127u) << 7) |
                             (((fine[2] >> lv) & 127u) << 14);
                    } else {
                        Coord c[3];
                        for (int a = 0; a < 3; ++a)
                            c[a] = kF32 ? coord_f32(__uint_as_float(w[a]))
                                        : coord_f64(__hiloint2double((int)w[2 * a + 1], (int)w[2 * a]));
                        uint32_t fx, fy, fz;
                        x = out_coord_frac<kF32>(c[0], op.ax[0], fx);
                        y = out_coord_frac<kF32>(c[1], op.ax[1], fy);
                        z = out_coord_frac<kF32>(c[2], op.ax[2], fz);
                        fw = pack_frac(fx, fy, fz);
                    }
                    if (x == kCoordError || y == kCoordError || z == kCoordError) set_error(err, kErrCoordRange);
                    nw[0] = (uint32_t)x;
                    nw[1] = (uint32_t)y;
                    nw[2] = (uint32_t)z;
                    nw[3] = (col & 0xFFu) | (((col >> 8) & 0xFFu) << 16);
                    nw[4] = (col >> 16) & 0xFFu;
                }
            }
            if (!image) {
                // each lane stores its own record with five stores (staging the
                // runs of a warp through shared memory for coalesced stores was
                // slower: 119.7M-point build 3.00 -> 2.73 ms)
                if (ok) {
                    lut[pos] = (uint32_t)(p0 + k);
                    frac[pos] = fw;
                    store_record_words(rec, pos, nw);
                }
            } else {
                if (ok) {
                    const uint32_t at = gs->at[slot], i = (at & 0xFFFFu) + rank;
                    gs->pos[i] = (uint32_t)pos;
                    gs->word[i] = fw;
                    gs->rec[i] = (uint16_t)k;
                    store_record_at(gs->image + (at >> 16) + rank * 18, nw);
                }
                __syncthreads();
                group_store(*gs, p0, lut, frac, rec);
            }
            if (group) {
                __syncthreads();
                group_clear(*gs);
                if (kMode == kByTile) __syncthreads();   // another round may follow
            }
        }
    });
}

// Copies byte range [src, src + bytes) to dst.  Both addresses are even (18-byte
// records); the body is written as aligned 16-byte stores assembled from
// 4-byte loads, realigned by a 16-bit funnel shift when needed.
__device__ __forceinline__ void copy_bytes_even(uint8_t* __restrict__ dst, const uint8_t* __restrict__ src,
                                                uint64_t bytes) {
    uintptr_t d0 = reinterpret_cast<uintptr_t>(dst), d1 = d0 + bytes;
    uintptr_t a0 = (d0 + 15) & ~(uintptr_t)15, a1 = d1 & ~(uintptr_t)15;
    const intptr_t delta = reinterpret_cast<intptr_t>(src) - (intptr_t)d0;
    if (a0 >= a1) {   // short range: 2-byte copies
        for (uintptr_t p = d0 + 2 * threadIdx.x; p < d1; p += 2 * blockDim.x)
            *reinterpret_cast<uint16_t*>(p) = *reinterpret_cast<const uint16_t*>(p + delta);
        return;
    }
    for (uintptr_t p = d0 + 2 * threadIdx.x; p < a0; p += 2 * blockDim.x)
        *reinterpret_cast<uint16_t*>(p) = *reinterpret_cast<const uint16_t*>(p + delta);
    for (uintptr_t p = a1 + 2 * threadIdx.x; p < d1; p += 2 * blockDim.x)
        *reinterpret_cast<uint16_t*>(p) = *reinterpret_cast<const uint16_t*>(p + delta);
    const uint64_t chunks = (a1 - a0) >> 4;
    for (uint64_t i = threadIdx.x; i < chunks; i += blockDim.x) {
        uintptr_t dp = a0 + i * 16, sp = dp + delta;
        const uint32_t* w = reinterpret_cast<const uint32_t*>(sp & ~(uintptr_t)3);
        uint4 o;
        if (sp & 2) {
            uint32_t w0 = w[0], w1 = w[1], w2 = w[2], w3 = w[3], w4 = w[4];
            o.x = __funnelshift_r(w0, w1, 16);
            o.y = __funnelshift_r(w1, w2, 16);
            o.z = __funnelshift_r(w2, w3, 16);
            o.w = __funnelshift_r(w3, w4, 16);
        } else {
            o.x = w[0];
            o.y = w[1];
            o.z = w[2];
            o.w = w[3];
        }
        *reinterpret_cast<uint4*>(dp) = o;
    }
}

__global__ void k_place(const uint64_t* __restrict__ src_off, const uint64_t* __restrict__ dst_off,
                        const uint32_t* __restrict__ count, uint32_t n_nodes, const uint8_t* __restrict__ stage_rec,
                        uint8_t* __restrict__ rec) {
    for (uint32_t v = blockIdx.x; v < n_nodes; v += gridDim.x)
        copy_bytes_even(rec + dst_off[v] * 18, stage_rec + src_off[v] * 18, (uint64_t)count[v] * 18);
}

// Output positions of the internal nodes: DFS post-order after the N leaf
// points (calculateWritingPosition, kernel_helpers.cuh:55-59).  One block
// scans the nodes' point counts in post-order (post[] lists internal indices)
// and writes the copy list of k_place; nothing is copied when an earlier stage
// reported a capacity error or the records exceed `cap`.
__global__ void __launch_bounds__(1024) k_place_prepare(const uint32_t* __restrict__ post, uint32_t n_internal,
                                                        const uint32_t* __restrict__ points,
                                                        const uint64_t* __restrict__ stage_off, uint64_t n,
                                                        uint64_t cap, uint64_t* src, uint64_t* dst, uint32_t* cnt,
                                                        uint64_t* node_dst, uint64_t* total, uint32_t* err) {
    __shared__ uint64_t warp_sums[32];
    const bool skip = *err != 0;   // (after any error levels may be without outputs)
    uint64_t running = 0;
    for (uint32_t k0 = 0; k0 < n_internal; k0 += blockDim.x) {
        const uint32_t k = k0 + threadIdx.x;
        const uint32_t ii = k < n_internal ? post[k] : 0;
        const uint64_t p = (k < n_internal && !skip) ? points[ii] : 0;
        uint64_t sum;
        const uint64_t pre = block_exclusive_scan64(p, warp_sums, sum);
        if (k < n_internal) {
            const uint64_t d = n + running + pre;
            src[k] = skip ? 0 : stage_off[ii];
            dst[k] = d;
            cnt[k] = (uint32_t)p;
            node_dst[ii] = d;
        }
        running += sum;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        *total = running;
        if (!skip && n + running > cap) atomicOr(err, kErrCapacity);
    }
    if (!skip && n + running > cap)   // nothing may be written past the record arrays
        for (uint32_t k = threadIdx.x; k < n_internal; k += blockDim.x) cnt[k] = 0;
}

// The words of the leaf records as distribution writes them, for a resident tree
// that is subsampled by the other kind of kernels: cell words (kCells) or
// sub-step words.  leaves: first record and level (kLeafLevelShift) of every
// leaf, in record order.  Gathers cloud points as k_place_units does.
template <bool kF32, bool kCells>
__global__ void __launch_bounds__(256) k_leaf_words(const uint8_t* __restrict__ cloud, uint64_t n, uint32_t stride,
                                                    const __grid_constant__ OutParams op,
                                                    const __grid_constant__ FixedGrid fg,
                                                    const uint64_t* __restrict__ leaves, uint32_t n_leaves,
                                                    const uint32_t* __restrict__ lut, uint32_t* __restrict__ word) {
    constexpr uint64_t kMask = (1ull << kLeafLevelShift) - 1;
    for (uint64_t pos = blockIdx.x * 256ull + threadIdx.x; pos < n; pos += gridDim.x * 256ull) {
        uint32_t lo = 0, hi = n_leaves;   // last leaf that starts at pos or before
        while (kCells && hi - lo > 1) {
            const uint32_t mid = (lo + hi) / 2;
            if ((leaves[mid] & kMask) <= pos) lo = mid;
            else hi = mid;
        }
        const uint8_t* rec = cloud + (uint64_t)lut[pos] * stride;
        uint32_t w[kF32 ? 4 : 7];
        gather_words<kF32, false>(rec, w);
        if (kCells) {
            const uint32_t lv = (uint32_t)(leaves[lo] >> kLeafLevelShift);
            uint32_t c[3], edge = 0;
            bool in = true;
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                uint64_t d;
                in &= fixed_difference(word_coord<kF32>(w, a), fg.ax[a].o, d);
                c[a] = fixed_cell(d, fg.ax[a].cell, fg.cells, edge);
            }
            if (!in) edge = 1u << 31;
            word[pos] = word_edge(edge) | ((c[0] >> lv) & 127u) | (((c[1] >> lv) & 127u) << 7) | (((c[2] >> lv) & 127u) << 14);
        } else {
            uint32_t f[3];
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                const Coord c = kF32 ? coord_f32(__uint_as_float(w[a]))
                                     : coord_f64(__hiloint2double((int)w[kF32 ? 0 : 2 * a + 1], (int)w[kF32 ? 0 : 2 * a]));
                out_coord_frac<kF32>(c, op.ax[a], f[a]);
            }
            word[pos] = pack_frac(f[0], f[1], f[2]);
        }
    }
}

__global__ void k_place_lut(const uint64_t* __restrict__ src_off, const uint64_t* __restrict__ dst_off,
                            const uint32_t* __restrict__ count, uint32_t n_nodes,
                            const uint32_t* __restrict__ stage_lut, uint32_t* __restrict__ lut) {
    for (uint32_t v = blockIdx.x; v < n_nodes; v += gridDim.x) {
        uint64_t s = src_off[v], d = dst_off[v];
        uint32_t c = count[v];
        for (uint32_t i = threadIdx.x; i < c; i += blockDim.x) lut[d + i] = stage_lut[s + i];
    }
}

}   // namespace

void allow_dynamic_smem(const void* kernel, size_t bytes) {
    static std::mutex mu;
    static std::map<std::pair<int, const void*>, size_t> limit;
    int dev = 0;
    cudaGetDevice(&dev);
    std::lock_guard<std::mutex> g(mu);
    size_t& cur = limit[{dev, kernel}];
    if (bytes <= cur) return;
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes) == cudaSuccess) cur = bytes;
    else cudaGetLastError();   // the launch reports the error
}

template <class Kernel>
static int chunk_grid_size(Kernel kernel, uint32_t threads, uint32_t tile, size_t smem, uint64_t n, int num_sms) {
    allow_dynamic_smem(reinterpret_cast<const void*>(kernel), smem);
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, smem) != cudaSuccess || per_sm < 1)
        per_sm = 1;
    const uint64_t tiles = (n + tile - 1) / tile;
    return (int)std::min<uint64_t>(tiles, (uint64_t)num_sms * per_sm);
}

int launch_count(const uint8_t* cloud, uint64_t n, uint32_t stride, bool float_input, const CloudGrid& g,
                  uint32_t* pyr0, uint8_t* occ, uint32_t* err, int num_sms, cudaStream_t stream) {
    if (n == 0) return 0;
    const size_t smem = chunk_smem(stride, g.grid, float_input, kCountTile).total;
    if (float_input) {
        const int grid = chunk_grid_size(k_count<true>, kCountThreads, kCountTile, smem, n, num_sms);
        k_count<true><<<grid, kCountThreads, smem, stream>>>(cloud, n, stride, g, pyr0, occ, err);
    } else {
        const int grid = chunk_grid_size(k_count<false>, kCountThreads, kCountTile, smem, n, num_sms);
        k_count<false><<<grid, kCountThreads, smem, stream>>>(cloud, n, stride, g, pyr0, occ, err);
    }
    return 1;
}

// Zeroes the 64-cell blocks of the finest level flagged in `occ`, and the
// flags: one thread per block.
__global__ void k_sparse_zero(uint32_t* __restrict__ pyr0, uint8_t* __restrict__ occ, uint64_t blocks) {
    const uint64_t b = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    if (b >= blocks || !occ[b]) return;
    uint4* d = reinterpret_cast<uint4*>(pyr0 + b * 64);
#pragma unroll
    for (int k = 0; k < 16; ++k) d[k] = make_uint4(0, 0, 0, 0);
    occ[b] = 0;
}

int launch_sparse_zero(uint32_t* pyr0, uint8_t* occ, uint64_t blocks, cudaStream_t stream) {
    if (!blocks) return 0;
    k_sparse_zero<<<(unsigned)((blocks + 255) / 256), 256, 0, stream>>>(pyr0, occ, blocks);
    return 1;
}

int launch_pyramid(uint32_t* pyr, const uint64_t* loff, uint32_t depth, uint32_t* nonzero, const uint8_t* occ,
                   cudaStream_t stream) {
    int launches = 0;
    for (uint32_t l = 0; l < top_level(depth); l += 2) {
        // level-(l+2) cells: (G0 >> (l+2))^3, the size of that level
        const uint64_t n2 = loff[l + 3] - loff[l + 2];
        if (l == 0 && occ)
            k_pyramid2_sparse<<<(unsigned)((n2 + 255) / 256), 256, 0, stream>>>(pyr, pyr + loff[1], pyr + loff[2], n2,
                                                                              nonzero, nonzero + 1, occ);
        else
            k_pyramid2<<<(unsigned)((n2 + kPyramidCells - 1) / kPyramidCells), 256, 0, stream>>>(
                pyr + loff[l], pyr + loff[l + 1], pyr + loff[l + 2], n2, nonzero + l, nonzero + l + 1);
        ++launches;
    }
    return launches;
}

int launch_enumerate(uint32_t* pyr, const uint64_t* loff_dev, uint32_t depth, uint32_t* nonzero, uint32_t threshold,
                     uint32_t* key, uint32_t* count, uint8_t* level, uint16_t* info, uint32_t* child_first,
                     uint32_t cap, uint32_t* level_start, uint32_t* n_nodes, uint32_t* err, cudaStream_t stream) {
    k_enumerate<<<1, 1024, 0, stream>>>(pyr, loff_dev, depth, top_level(depth), nonzero, threshold, key, count, level,
                                        info, child_first, cap, level_start, n_nodes, err);
    return 1;
}

int launch_bbox(const uint8_t* cloud, uint64_t n, uint32_t stride, bool float_input, long long* keys, int num_sms,
                cudaStream_t stream) {
    k_bbox_init<<<1, 32, 0, stream>>>(keys);
    const uint64_t want = (n + 255) / 256;
    const unsigned grid = (unsigned)std::max<uint64_t>(1, std::min<uint64_t>(want, (uint64_t)num_sms * 8));
    if (float_input) k_bbox<true><<<grid, 256, 0, stream>>>(cloud, n, stride, keys);
    else k_bbox<false><<<grid, 256, 0, stream>>>(cloud, n, stride, keys);
    return 2;
}

int launch_leaf_prep(const uint32_t* n_nodes, const uint16_t* info, const uint32_t* count, const uint8_t* level,
                     const uint32_t* key, uint32_t* pyr, const uint64_t* loff_dev, uint64_t* data_idx, uint32_t* fill,
                     uint64_t n_points, uint32_t* err, cudaStream_t stream) {
    k_leaf_prep<<<1, 1024, 0, stream>>>(n_nodes, info, count, level, key, pyr, loff_dev, data_idx, fill, n_points, err);
    return 1;
}

int launch_leaf_words(const uint8_t* cloud, uint64_t n, uint32_t stride, bool float_input, bool cells,
                      const OutParams& out, const FixedGrid& fixed, const uint64_t* leaves, uint32_t n_leaves,
                      const uint32_t* lut, uint32_t* word, int num_sms, cudaStream_t stream) {
    if (!n) return 0;
    const unsigned grid = (unsigned)std::max<uint64_t>(1, std::min<uint64_t>((n + 255) / 256, (uint64_t)num_sms * 8));
    const auto go = float_input ? cells ? k_leaf_words<true, true> : k_leaf_words<true, false>
                                : cells ? k_leaf_words<false, true> : k_leaf_words<false, false>;
    go<<<grid, 256, 0, stream>>>(cloud, n, stride, out, fixed, leaves, n_leaves, lut, word);
    return 1;
}

int launch_push_tags(uint32_t* pyr, const uint64_t* loff_dev, uint32_t depth, const uint8_t* occ, uint32_t* err,
                     const uint8_t* cloud, uint64_t n, uint32_t stride, bool float_input, const CloudGrid& g,
                     cudaStream_t stream) {
    const uint64_t n1 = (uint64_t)(g.grid / 2) * (g.grid / 2) * (g.grid / 2);
    if (!n1) return 0;
    const uint32_t blocks = (uint32_t)((n1 + 255) / 256);
    k_push_tags<<<blocks + kOrderWarps / 8, 256, 0, stream>>>(pyr, loff_dev, depth, n1, occ, err, cloud, n, stride,
                                                              float_input, g, blocks);
    return 1;
}

namespace {

template <bool kF32, bool kCells, int kMode>
void distribute_on(const uint8_t* cloud, uint64_t n, uint32_t stride, const CloudGrid& g, const OutParams& out,
                   const FixedGrid& fg, const uint32_t* pyr0, const uint64_t* data_idx, uint32_t* fill, uint32_t* lut,
                   uint8_t* rec, uint32_t* word, uint32_t* err, const uint32_t* order, int num_sms,
                   cudaStream_t stream) {
    constexpr uint32_t kTile = dist_tile(kMode), kThreads = dist_threads(kMode);
    const size_t smem = align_up(chunk_smem(stride, g.grid, kF32, kTile, !kCells).total, 16) +
                        (kMode != kDirect ? sizeof(GroupSmem<kMode>) : 0);
    const int grid = chunk_grid_size(k_distribute<kF32, kCells, kMode>, kThreads, kTile, smem, n, num_sms);
    k_distribute<kF32, kCells, kMode><<<grid, kThreads, smem, stream>>>(cloud, n, stride, g, out, fg, pyr0, data_idx,
                                                                         fill, lut, rec, word, err, order);
}

}   // namespace

int launch_distribute(const uint8_t* cloud, uint64_t n, uint32_t stride, bool float_input, const CloudGrid& g,
                      const OutParams& out, const uint32_t* pyr0, const uint64_t* data_idx, uint32_t* fill,
                      uint32_t* lut, uint8_t* rec, uint32_t* frac, uint32_t* err, int num_sms,
                      cudaStream_t stream) {
    if (n == 0) return 0;
    const auto go = float_input ? distribute_on<true, false, kDirect> : distribute_on<false, false, kDirect>;
    go(cloud, n, stride, g, out, FixedGrid{}, pyr0, data_idx, fill, lut, rec, frac, err, nullptr, num_sms, stream);
    return 1;
}

int launch_distribute_cells(const uint8_t* cloud, uint64_t n, uint32_t stride, bool float_input, const CloudGrid& g,
                            const OutParams& out, const FixedGrid& fixed, const uint32_t* pyr0,
                            const uint64_t* data_idx, uint32_t* fill, uint32_t* lut, uint8_t* rec, uint32_t* word,
                            uint32_t* err, int num_sms, cudaStream_t stream) {
    if (n == 0) return 0;
    // records too long for the grouped kernels' shared memory are stored lane
    // by lane; on a small cloud the second launch costs more than it can give
    const bool fits = stride <= kGroupMaxStride, both = fits && n >= kGroupMinPoints;
    const uint32_t* order = both ? err + kOrderWord : nullptr;
    const auto by_lane = !float_input ? distribute_on<false, true, kDirect>
                         : fits       ? distribute_on<true, true, kByTile>
                                      : distribute_on<true, true, kDirect>;
    by_lane(cloud, n, stride, g, out, fixed, pyr0, data_idx, fill, lut, rec, word, err, order, num_sms, stream);
    if (!both) return 1;
    const auto grouped = float_input ? distribute_on<true, true, kGrouped> : distribute_on<false, true, kGrouped>;
    grouped(cloud, n, stride, g, out, fixed, pyr0, data_idx, fill, lut, rec, word, err, order, num_sms, stream);
    return 2;
}

int launch_place(const uint64_t* src_off, const uint64_t* dst_off, const uint32_t* count, uint32_t n_nodes,
                 const uint8_t* stage_rec, uint8_t* rec, cudaStream_t stream) {
    if (!n_nodes) return 0;
    unsigned grid = n_nodes < 8192 ? n_nodes : 8192;
    k_place<<<grid, 256, 0, stream>>>(src_off, dst_off, count, n_nodes, stage_rec, rec);
    return 1;
}

int launch_place_prepare(const uint32_t* post, uint32_t n_internal, const uint32_t* points, const uint64_t* stage_off,
                         uint64_t n, uint64_t cap, uint64_t* src, uint64_t* dst, uint32_t* cnt, uint64_t* node_dst,
                         uint64_t* total, uint32_t* err, cudaStream_t stream) {
    k_place_prepare<<<1, 1024, 0, stream>>>(post, n_internal, points, stage_off, n, cap, src, dst, cnt, node_dst, total,
                                            err);
    return 1;
}

int launch_place_lut(const uint64_t* src_off, const uint64_t* dst_off, const uint32_t* count, uint32_t n_nodes,
                     const uint32_t* stage_lut, uint32_t* lut, cudaStream_t stream) {
    if (!n_nodes) return 0;
    unsigned grid = n_nodes < 8192 ? n_nodes : 8192;
    k_place_lut<<<grid, 256, 0, stream>>>(src_off, dst_off, count, n_nodes, stage_lut, lut);
    return 1;
}

}   // namespace oc
