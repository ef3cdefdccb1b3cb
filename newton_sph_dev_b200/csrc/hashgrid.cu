// hashgrid.cu — HashGrid build (hash + stable LSD radix sort + cell ranges)
// and the batched Warp-order query.
//
// Replaces wp.HashGrid (external warp-lang 1.14.0.dev20260511), constructed
// at newton/_src/sim/builder.py:9853, reserved at
// newton/_src/solvers/xpbd/solver_xpbd.py:139 and built at
// solver_xpbd.py:315-319; its device query is used at
// newton/_src/solvers/semi_implicit/kernels_contact.py:54,68,71.
//
// Build pipeline (all stream-ordered, no allocation, no host sync):
//   k_hash_hist   original order: cell id per point + digit-0 tile histograms;
//                 also clears the cell ranges the previous build wrote.
//   per 8-bit digit pass: [k_upsweep] -> k_scan_rows -> k_downsweep
//                 stable multi-split per tile of 256 x kItems keys (2048,
//                 or 512 for builds of at most kSmallBuildPoints points, so
//                 that small builds still spread over the SMs; the sorted
//                 result does not depend on the tile) (warp match_any ranks,
//                 shared-memory staging for coalesced scatter). The last pass
//                 writes point_cells / point_ids and, in SPH mode, gathers the
//                 sorted float4 mirrors of position and velocity.
//   k_ranges      cell_starts / cell_ends from the sorted cell ids.
// Single-world grids whose table holds at most kCountCellsPerPoint cells per
// point (the SPH solver's grids) build by cell counts instead (count_build:
// atomic counts, per-tile sums and a scan of the cell table that writes the
// ranges, scatter, stable rank within each cell): 5 launches instead of 10,
// the same result. Builds of at most kRankMax points count comparisons instead
// (k_rank_cells, k_rank_build): 2 launches, the same result.
#include <algorithm>
#include <cstdio>
#include <mutex>
#include <string>
#include <vector>

#include "nsph_internal.cuh"

namespace nsph {

NSPH_BOUNDS_READER(hashgrid)

namespace {

__device__ __forceinline__ unsigned lanemask_lt()
{
    unsigned m;
    asm volatile("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}

// the sorted mirrors of particle p
__device__ __forceinline__ void mirrors_of(const GatherArgs& gather, int p, float4& xs, float4& vs)
{
    const size_t i = (size_t)p;
    const Row3 x = load_row(gather.x + 3 * i), v = load_row(gather.v + 3 * i);
    const int fl = gather.flags[i];
    const bool active = (fl & NSPH_PARTICLE_ACTIVE) != 0;
    const float m = gather.mass[i];
    const float w = gather.inv_mass[i];
    int gw = gather.world ? gather.world[i] : 0;
    gw = gw < 0 ? 0 : (gw >= gather.world_count ? gather.world_count - 1 : gw);
    const int attr = (active ? kAttrActive : 0) | (w > 0.f ? kAttrDynamic : 0) | (gw << kAttrGravShift);
    xs = make_float4(x.x, x.y, x.z, mirror_mass(m, active));
    vs = make_float4(v.x, v.y, v.z, __int_as_float(attr));
}

__device__ __forceinline__ void gather_particle(const GatherArgs& gather, int p, int g)
{
    float4 xs, vs;
    mirrors_of(gather, p, xs, vs);
    gather.xs[g] = xs;
    gather.vs[g] = vs;
}

// the cell of point idx, in its world's part of the table; sets bad for a
// position that is not finite
__device__ __forceinline__ int cell_of_point(const float* __restrict__ points, int idx, float inv, int dx, int dy,
                                             int dz, const int* __restrict__ world,
                                             const WorldCells* __restrict__ wcells, int world_count, bool& bad)
{
    const float x = points[3 * (size_t)idx + 0];
    const float y = points[3 * (size_t)idx + 1];
    const float z = points[3 * (size_t)idx + 2];
    bad |= !(isfinite(x) && isfinite(y) && isfinite(z));
    if (!wcells) return point_cell(x, y, z, inv, dx, dy, dz);
    int w = world ? world[idx] : 0;
    w = w < 0 ? 0 : (w >= world_count ? world_count - 1 : w);
    const WorldCells c = wcells[w];
    return (int)(c.off + point_cell(x, y, z, c.inv, c.dx, c.dy, c.dz));
}

// --------------------------------------------------------------------------
// k_hash_hist: keys/vals in original order + histogram of digit 0 per tile.
// Also clears the previous build's occupied cells (their first sorted entry
// resets start/end to 0), so no full memset of the cell tables is needed.
// --------------------------------------------------------------------------
template <int kItems>
__global__ void __launch_bounds__(kSortThreads) k_hash_hist(
    const float* __restrict__ points, int n, float inv, int dx, int dy, int dz, int* __restrict__ keys,
    int* __restrict__ vals, unsigned* __restrict__ hist, int ntiles, int digit_mask,
    const int* __restrict__ prev_cells, int prev_n, int2* __restrict__ ranges, unsigned* __restrict__ status,
    const int* __restrict__ world, const WorldCells* __restrict__ wcells, int world_count)
{
    launch_entry();
    __shared__ unsigned wh[kSortThreads / 32][kRadix];
    const int warp = threadIdx.x >> 5;
    for (int i = threadIdx.x; i < (kSortThreads / 32) * kRadix; i += kSortThreads) (&wh[0][0])[i] = 0u;
    __syncthreads();

    const int base = blockIdx.x * (kSortThreads * kItems);
    bool bad = false;
#pragma unroll 4
    for (int it = 0; it < kItems; ++it) {
        const int idx = base + it * kSortThreads + threadIdx.x;
        if (idx < prev_n) {
            const int c = prev_cells[idx];
            if (idx == 0 || prev_cells[idx - 1] != c) ranges[c] = make_int2(0, 0);
        }
        if (idx < n) {
            const int key = cell_of_point(points, idx, inv, dx, dy, dz, world, wcells, world_count, bad);
            keys[idx] = key;
            vals[idx] = idx;
            atomicAdd(&wh[warp][key & digit_mask], 1u);
        }
    }
    if (bad && status) atomicOr(status, (unsigned)NSPH_STATUS_NONFINITE_INPUT);
    __syncthreads();
    if (blockIdx.x < ntiles) {
        for (int d = threadIdx.x; d < kRadix; d += kSortThreads) {
            unsigned s = 0;
#pragma unroll
            for (int w = 0; w < kSortThreads / 32; ++w) s += wh[w][d];
            hist[(size_t)d * ntiles + blockIdx.x] = s;
        }
    }
}

// Histogram of one digit per tile (passes after the first).
template <int kItems>
__global__ void __launch_bounds__(kSortThreads) k_upsweep(const int* __restrict__ keys, int n, int shift,
                                                          int digit_mask, unsigned* __restrict__ hist,
                                                          int ntiles)
{
    launch_entry();
    __shared__ unsigned wh[kSortThreads / 32][kRadix];
    const int warp = threadIdx.x >> 5;
    for (int i = threadIdx.x; i < (kSortThreads / 32) * kRadix; i += kSortThreads) (&wh[0][0])[i] = 0u;
    __syncthreads();
    const int base = blockIdx.x * (kSortThreads * kItems);
#pragma unroll 4
    for (int it = 0; it < kItems; ++it) {
        const int idx = base + it * kSortThreads + threadIdx.x;
        if (idx < n) atomicAdd(&wh[warp][(keys[idx] >> shift) & digit_mask], 1u);
    }
    __syncthreads();
    for (int d = threadIdx.x; d < kRadix; d += kSortThreads) {
        unsigned s = 0;
#pragma unroll
        for (int w = 0; w < kSortThreads / 32; ++w) s += wh[w][d];
        hist[(size_t)d * ntiles + blockIdx.x] = s;
    }
}

// Row scan of the digit-major histogram table: CTA d turns hist[d][0..ntiles)
// into exclusive offsets within digit d and writes the digit's total to
// digit_tot[d]. The downsweep adds the exclusive scan of the digit totals.
constexpr int kScanThreads = 256;
__device__ __forceinline__ unsigned block_exclusive_scan(unsigned v, unsigned& total, unsigned* ws)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += t;
    }
    if (lane == 31) ws[warp] = incl;
    __syncthreads();
    unsigned base = 0, tot = 0;
#pragma unroll
    for (int w = 0; w < kScanThreads / 32; ++w) {
        const unsigned x = ws[w];
        base += (w < warp) ? x : 0u;
        tot += x;
    }
    __syncthreads();  // ws reusable after return
    total = tot;
    return base + incl - v;
}

__global__ void __launch_bounds__(kScanThreads) k_scan_rows(unsigned* __restrict__ hist, int ntiles,
                                                            unsigned* __restrict__ digit_tot)
{
    launch_entry();
    __shared__ unsigned ws[kScanThreads / 32];
    unsigned* row = hist + (size_t)blockIdx.x * ntiles;
    unsigned carry = 0;
    for (int base = 0; base < ntiles; base += kScanThreads) {
        const int i = base + threadIdx.x;
        const unsigned v = i < ntiles ? row[i] : 0u;
        unsigned tot;
        const unsigned ex = block_exclusive_scan(v, tot, ws);
        if (i < ntiles) row[i] = carry + ex;
        carry += tot;
    }
    if (threadIdx.x == 0) digit_tot[blockIdx.x] = carry;
}

// --------------------------------------------------------------------------
// k_downsweep: stable scatter of one digit pass.
// Warp w owns tile elements [w*32*kItems, (w+1)*32*kItems) in kItems rounds
// of 32; within a round lanes with equal digits are ranked by __match_any_sync, and a
// per-warp counter carries ranks across rounds, so the order inside a tile
// is exactly the input order per digit. Keys are staged in shared memory in
// tile-sorted order and written out in runs (coalesced).
// --------------------------------------------------------------------------
constexpr int kWarps = kSortThreads / 32;

template <int kItems>
struct DownsweepSmem {
    unsigned warp_cnt[kWarps][kRadix];
    unsigned tile_off[kRadix];
    unsigned glob_off[kRadix];
    int keys[kSortThreads * kItems];
    int vals[kSortThreads * kItems];
};

template <bool kGather, int kItems>
__global__ void __launch_bounds__(kSortThreads) k_downsweep(const int* __restrict__ keys_in,
                                                            const int* __restrict__ vals_in,
                                                            int* __restrict__ keys_out, int* __restrict__ vals_out,
                                                            int n, int shift, int digit_mask,
                                                            const unsigned* __restrict__ hist, int ntiles,
                                                            const unsigned* __restrict__ digit_tot,
                                                            GatherArgs gather)
{
    launch_entry();
    constexpr int kTile = kSortThreads * kItems;
    constexpr int kPerWarp = kTile / kWarps;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    DownsweepSmem<kItems>& sm = *reinterpret_cast<DownsweepSmem<kItems>*>(smem_raw);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int i = threadIdx.x; i < kWarps * kRadix; i += kSortThreads) (&sm.warp_cnt[0][0])[i] = 0u;
    __syncthreads();

    const int tile_base = blockIdx.x * kTile;
    const int tile_n = min(kTile, n - tile_base);
    int key[kItems], val[kItems];
    unsigned rank[kItems];
    const unsigned lt = lanemask_lt();
#pragma unroll
    for (int r = 0; r < kItems; ++r) {
        const int local = warp * kPerWarp + r * 32 + lane;
        const bool valid = local < tile_n;
        key[r] = valid ? keys_in[tile_base + local] : 0;
        val[r] = valid ? vals_in[tile_base + local] : 0;
        const int d = valid ? ((key[r] >> shift) & digit_mask) : kRadix;  // kRadix: sentinel group
        const unsigned peers = __match_any_sync(0xffffffffu, d);
        const unsigned before = __popc(peers & lt);
        unsigned base = 0;
        if (valid) base = sm.warp_cnt[warp][d];
        __syncwarp();
        if (valid && before == 0) sm.warp_cnt[warp][d] = base + __popc(peers);
        __syncwarp();
        rank[r] = base + before;
    }
    __syncthreads();
    // per digit (thread d): exclusive prefix over warps and this tile's total
    const int d = threadIdx.x;  // kRadix == kSortThreads
    unsigned total = 0;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) {
        const unsigned c = sm.warp_cnt[w][d];
        sm.warp_cnt[w][d] = total;
        total += c;
    }
    __shared__ unsigned ws[kWarps];
    unsigned dummy;
    // global offset of digit d from this tile: digits before d (all tiles) +
    // digit d in the tiles before this one
    const unsigned dbase = block_exclusive_scan(digit_tot[d], dummy, ws);
    sm.glob_off[d] = dbase + hist[(size_t)d * ntiles + blockIdx.x];
    // exclusive scan of this tile's digit totals
    sm.tile_off[d] = block_exclusive_scan(total, dummy, ws);
    __syncthreads();
#pragma unroll
    for (int r = 0; r < kItems; ++r) {
        const int local = warp * kPerWarp + r * 32 + lane;
        if (local < tile_n) {
            const int d = (key[r] >> shift) & digit_mask;
            const unsigned pos = sm.tile_off[d] + sm.warp_cnt[warp][d] + rank[r];
            sm.keys[pos] = key[r];
            sm.vals[pos] = val[r];
        }
    }
    __syncthreads();
    for (int p = threadIdx.x; p < tile_n; p += kSortThreads) {
        const int k = sm.keys[p];
        const int v = sm.vals[p];
        const int d = (k >> shift) & digit_mask;
        const unsigned g = sm.glob_off[d] + (unsigned)p - sm.tile_off[d];
        keys_out[g] = k;
        vals_out[g] = v;
        if constexpr (kGather) {
            gather_particle(gather, v, (int)g);
        }
    }
}

// Cell [start, end) ranges from sorted cell ids (Warp's compute_cell_offsets
// semantics; cells not written keep the {0,0} of an empty cell).
__global__ void k_ranges(const int* __restrict__ cells, int n, int2* __restrict__ ranges)
{
    launch_entry();
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const int c = cells[k];
    int* r = reinterpret_cast<int*>(ranges + c);
    if (k == 0 || cells[k - 1] != c) r[0] = k;
    if (k == n - 1 || cells[k + 1] != c) r[1] = k + 1;
}

// --------------------------------------------------------------------------
// Counting build (single-world grids whose cell table is at most a few times
// the point count): the stable (cell, index) order from cell counts instead
// of three radix passes.
//   k_cc_count        cell of each point (original order), its slot in the
//                     cell from an atomic counter (an arbitrary order within a
//                     cell); clears the ranges of the previous build's cells
//   k_cc_tile_sums    the points of each tile of kCsTile cells
//   k_cc_scan_ranges  per tile: its offset (the sum of the earlier tiles'
//                     counts), the exclusive scan of its cells' counts, the
//                     ranges of its occupied cells
//   k_cc_scatter      point -> start + slot (the arbitrary order), with its cell
//   k_cc_rank         per cell-ordered position: its point goes to start +
//                     (points of its cell with a smaller index), the stable
//                     order; writes point_cells / point_ids, gathers the
//                     sorted mirrors in SPH mode, and zeroes the cell's count
// No kernel waits on another block. The result is identical to the stable
// radix sort's.
// --------------------------------------------------------------------------
constexpr int kCsThreads = 256;  // k_cc_scan_ranges
constexpr int kCsPer = 32;       // cells per thread
constexpr int kCsTile = kCsThreads * kCsPer;

__global__ void __launch_bounds__(256) k_cc_count(const float* __restrict__ points, int n, float inv, int dx, int dy,
                                                  int dz, int* __restrict__ count, int* __restrict__ cells,
                                                  int* __restrict__ slots, const int* __restrict__ prev_cells,
                                                  int prev_n, int2* __restrict__ ranges,
                                                  unsigned* __restrict__ status)
{
    launch_entry();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    // the previous build's cells: the first sorted entry of each clears its range
    for (int k = i; k < prev_n; k += gridDim.x * blockDim.x) {
        const int c = prev_cells[k];
        if (k == 0 || prev_cells[k - 1] != c) ranges[c] = make_int2(0, 0);
    }
    bool bad = false;
    if (i < n) {
        const float x = points[3 * (size_t)i + 0];
        const float y = points[3 * (size_t)i + 1];
        const float z = points[3 * (size_t)i + 2];
        bad = !(isfinite(x) && isfinite(y) && isfinite(z));
        const int c = point_cell(x, y, z, inv, dx, dy, dz);
        cells[i] = c;
        slots[i] = atomicAdd(count + c, 1);
    }
    if (bad && status) atomicOr(status, (unsigned)NSPH_STATUS_NONFINITE_INPUT);
}

// The counts of a tile by warp: each takes a segment of kCsSegment consecutive
// cells, lane l the cells 4 l .. 4 l + 3 of each of its kCsQuads groups of 128,
// so that a warp's loads are contiguous (32 cells in a row per thread had
// every load touch 32 lines: 20.5 -> 11.4 us for both kernels on the 4.2M cells
// of the 1M tank).
constexpr int kCsQuads = kCsPer / 4;
constexpr int kCsSegment = 32 * kCsPer;

__device__ __forceinline__ void cc_load_counts(const int* __restrict__ count, long long ncells, long long c0,
                                               int lane, int4 (&v)[kCsQuads])
{
    const long long c = c0 + 4 * lane;
    if (c0 + kCsSegment <= ncells) {  // count is 256-byte aligned and c0 a multiple of kCsSegment
        const int4* p4 = reinterpret_cast<const int4*>(count + c);
#pragma unroll
        for (int q = 0; q < kCsQuads; ++q) v[q] = p4[32 * q];
    } else {
#pragma unroll
        for (int q = 0; q < kCsQuads; ++q) {
            const long long cq = c + 128 * q;
            v[q] = make_int4(cq < ncells ? count[cq] : 0, cq + 1 < ncells ? count[cq + 1] : 0,
                             cq + 2 < ncells ? count[cq + 2] : 0, cq + 3 < ncells ? count[cq + 3] : 0);
        }
    }
}

__global__ void __launch_bounds__(kCsThreads) k_cc_tile_sums(const int* __restrict__ count, long long ncells,
                                                             int* __restrict__ tile_count)
{
    launch_entry();
    __shared__ int part[kCsThreads / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int4 v[kCsQuads];
    cc_load_counts(count, ncells, (long long)blockIdx.x * kCsTile + (long long)warp * kCsSegment, lane, v);
    int sum = 0;
#pragma unroll
    for (int q = 0; q < kCsQuads; ++q) sum += v[q].x + v[q].y + v[q].z + v[q].w;
    sum = __reduce_add_sync(0xffffffffu, sum);
    if (lane == 0) part[warp] = sum;
    __syncthreads();
    if (threadIdx.x == 0) {
        int total = 0;
#pragma unroll
        for (int w = 0; w < kCsThreads / 32; ++w) total += part[w];
        tile_count[blockIdx.x] = total;
    }
}

__global__ void __launch_bounds__(kCsThreads) k_cc_scan_ranges(const int* __restrict__ count,
                                                               const int* __restrict__ tile_count, long long ncells,
                                                               int2* __restrict__ ranges)
{
    launch_entry();
    __shared__ int ws[kCsThreads / 32];
    __shared__ int s_base[kCsThreads / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int tile = blockIdx.x;
    const long long c0 = (long long)tile * kCsTile + (long long)warp * kCsSegment;
    int4 v[kCsQuads];
    cc_load_counts(count, ncells, c0, lane, v);
    // the tile's offset: the counts of the tiles before it
    int before = 0;
    for (int q = threadIdx.x; q < tile; q += kCsThreads) before += tile_count[q];
    int sum = 0;
#pragma unroll
    for (int q = 0; q < kCsQuads; ++q) sum += v[q].x + v[q].y + v[q].z + v[q].w;
    sum = __reduce_add_sync(0xffffffffu, sum);
    before = __reduce_add_sync(0xffffffffu, before);
    if (lane == 0) {
        ws[warp] = sum;
        s_base[warp] = before;
    }
    __syncthreads();
    if (sum == 0) return;  // the segment is empty (its cells keep {0, 0})
    int start = 0;
#pragma unroll
    for (int w = 0; w < kCsThreads / 32; ++w) start += s_base[w] + (w < warp ? ws[w] : 0);
#pragma unroll
    for (int q = 0; q < kCsQuads; ++q) {
        const int mine = v[q].x + v[q].y + v[q].z + v[q].w;
        int inc = mine;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += y;
        }
        int at = start + inc - mine;
        int2* r = ranges + c0 + 128 * q + 4 * lane;
        if (v[q].x) r[0] = make_int2(at, at + v[q].x);  // empty cells keep {0, 0}
        at += v[q].x;
        if (v[q].y) r[1] = make_int2(at, at + v[q].y);
        at += v[q].y;
        if (v[q].z) r[2] = make_int2(at, at + v[q].z);
        at += v[q].z;
        if (v[q].w) r[3] = make_int2(at, at + v[q].w);
        start += __shfl_sync(0xffffffffu, inc, 31);
    }
}

__global__ void __launch_bounds__(256) k_cc_scatter(const int* __restrict__ cells, const int* __restrict__ slots,
                                                    const int2* __restrict__ ranges, int n, int* __restrict__ tmp,
                                                    int* __restrict__ tmp_cells)
{
    launch_entry();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int c = cells[i], at = ranges[c].x + slots[i];
    if (in_bounds(at >= 0 && at < n)) {
        tmp[at] = i;
        tmp_cells[at] = c;
    }
}

// one thread per position q of the cell-ordered (not yet stable) array: its
// point i, the rank of i among its cell's points, and the stable position
// start + rank, which lies in the same cell's range, so neighbouring threads
// write neighbouring positions
__global__ void __launch_bounds__(256) k_cc_rank(const int* __restrict__ tmp_cells, const int2* __restrict__ ranges,
                                                 const int* __restrict__ tmp, int n, int* __restrict__ count,
                                                 int* __restrict__ point_cells, int* __restrict__ point_ids,
                                                 GatherArgs gather, bool do_gather)
{
    launch_entry();
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= n) return;
    const int i = tmp[q];
    const int c = tmp_cells[q];
    if (!in_bounds(i >= 0 && i < n)) return;
    float4 xs, vs;
    if (do_gather) mirrors_of(gather, i, xs, vs);  // the gathered loads go out before the rank loop
    const int2 se = ranges[c];
    if (!in_bounds(se.x >= 0 && se.x <= q && q < se.y && se.y <= n)) return;
    int rank = 0;
    for (int t = se.x; t < se.y; ++t) rank += tmp[t] < i;
    if (rank == 0) count[c] = 0;  // the counts start at zero for the next build
    const int g = se.x + rank;
    point_cells[g] = c;
    point_ids[g] = i;
    if (do_gather) {
        gather.xs[g] = xs;
        gather.vs[g] = vs;
    }
}

// --------------------------------------------------------------------------
// Builds of a few thousand points in two launches: k_rank_cells writes the
// cell of each point (and clears the previous build's cells), k_rank_build
// counts, for each point, the points of smaller cells and those of its own:
// the counts are the point's place in the stable order and its cell's range.
// n^2 comparisons, but in one pass; such a build is bound by its launches (five
// of the counting build, ten of the radix sort). Whole step on
// a B200, with this build and without: 23 us and 27 (counting) or 38 (radix) at
// 1,000 particles, 25 and 28 or 39 at 2,197, 28 and 29.5 or 42 at 4,096; at
// 8,000 it loses (build phase 24 us, counting 16). A bitonic sort in one block
// took 46 us at 2,197.
// --------------------------------------------------------------------------
constexpr int kRankThreads = 256;
constexpr int kRankPoints = 2;           // per warp
constexpr int kRankMax = 4096;           // points
constexpr int kRankPrev = 65536;         // points of the previous build whose cells it clears

__global__ void __launch_bounds__(kRankThreads) k_rank_cells(
    const float* __restrict__ points, int n, float inv, int dx, int dy, int dz, int* __restrict__ keys,
    const int* __restrict__ prev_cells, int prev_n, int2* __restrict__ ranges, unsigned* __restrict__ status,
    const int* __restrict__ world, const WorldCells* __restrict__ wcells, int world_count)
{
    launch_entry();
    const int idx = blockIdx.x * kRankThreads + threadIdx.x;
    if (idx < prev_n) {
        const int c = prev_cells[idx];
        if (idx == 0 || prev_cells[idx - 1] != c) ranges[c] = make_int2(0, 0);
    }
    bool bad = false;
    if (idx < n) keys[idx] = cell_of_point(points, idx, inv, dx, dy, dz, world, wcells, world_count, bad);
    if (bad && status) atomicOr(status, (unsigned)NSPH_STATUS_NONFINITE_INPUT);
}

__global__ void __launch_bounds__(kRankThreads) k_rank_build(const int* __restrict__ keys, int n,
                                                             int2* __restrict__ ranges,
                                                             int* __restrict__ point_cells,
                                                             int* __restrict__ point_ids, GatherArgs gather,
                                                             bool do_gather)
{
    launch_entry();
    const int lane = threadIdx.x & 31;
    const int i0 = (blockIdx.x * (kRankThreads / 32) + (threadIdx.x >> 5)) * kRankPoints;
    if (i0 >= n) return;
    int c[kRankPoints], less[kRankPoints], same[kRankPoints], before[kRankPoints];
#pragma unroll
    for (int p = 0; p < kRankPoints; ++p) {
        c[p] = i0 + p < n ? keys[i0 + p] : 0;
        less[p] = same[p] = before[p] = 0;
    }
    auto count_same = [&](int k, int j) {
#pragma unroll
        for (int p = 0; p < kRankPoints; ++p) {
            same[p] += k == c[p];
            before[p] += (k == c[p]) & (j < i0 + p);
        }
    };
    const int whole = n & ~3;
#pragma unroll 4
    for (int j = 4 * lane; j < whole; j += 128) {
        const int4 k4 = *reinterpret_cast<const int4*>(keys + j);
        const int k[4] = {k4.x, k4.y, k4.z, k4.w};
        bool any = false;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
#pragma unroll
            for (int p = 0; p < kRankPoints; ++p) {
                less[p] += k[u] < c[p];
                any |= k[u] == c[p];
            }
        }
        if (any) {
#pragma unroll
            for (int u = 0; u < 4; ++u) count_same(k[u], j + u);
        }
    }
    if (whole + lane < n) {
        const int k = keys[whole + lane];
#pragma unroll
        for (int p = 0; p < kRankPoints; ++p) less[p] += k < c[p];
        count_same(k, whole + lane);
    }
#pragma unroll
    for (int p = 0; p < kRankPoints; ++p) {
        less[p] = __reduce_add_sync(0xffffffffu, less[p]);
        same[p] = __reduce_add_sync(0xffffffffu, same[p]);
        before[p] = __reduce_add_sync(0xffffffffu, before[p]);
    }
#pragma unroll
    for (int p = 0; p < kRankPoints; ++p) {
        if (lane != p || i0 + p >= n) continue;
        const int place = less[p] + before[p];
        point_cells[place] = c[p];
        point_ids[place] = i0 + p;
        ranges[c[p]] = make_int2(less[p], less[p] + same[p]);  // the same from every point of the cell
        if (do_gather) gather_particle(gather, i0 + p, place);
    }
}

// Batched Warp-order query: counts, or ids at offsets. kQueryLanes lanes per
// query: lane r takes the box's rows r, r + kQueryLanes, .. (a row's cells
// are one run of sorted positions), whose places in the answer follow from a
// prefix sum over the rows. One thread per query walked its 27 cells and wrote
// its candidates one after another (300,007 points, 40,001 queries of 31
// candidates: count 15 us, fill 35 us; the whole build-and-query call 124 -> 111 us). Clamped boxes, rows that
// wrap in x and boxes of more than two rows per lane are walked by one lane.
constexpr int kQueryLanes = 8;

__global__ void __launch_bounds__(128) k_query(const __grid_constant__ GridDev g, const float* __restrict__ q, int nq,
                                               float radius, int* __restrict__ counts,
                                               const long long* __restrict__ offsets, int* __restrict__ out)
{
    launch_entry();
    constexpr unsigned kAll = 0xffffffffu;
    const long long thread = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const int sub = threadIdx.x & (kQueryLanes - 1);
    const bool live = thread / kQueryLanes < nq;
    const int t = live ? (int)(thread / kQueryLanes) : nq - 1;
    const float px = q[3 * (size_t)t], py = q[3 * (size_t)t + 1], pz = q[3 * (size_t)t + 2];
    int xl, xh, yl, yh, zl, zh;
    bool clamped = false;
    box_axis_regular(px, radius, g.inv, g.dx, xl, xh, clamped);
    box_axis_regular(py, radius, g.inv, g.dy, yl, yh, clamped);
    box_axis_regular(pz, radius, g.inv, g.dz, zl, zh, clamped);
    const int nx = xh - xl + 1, ny = yh - yl + 1;
    const long long rows = (long long)ny * (zh - zl + 1);
    const int cx = clamped ? 0 : wrap_cell(xl, g.dx);
    const bool by_rows = !clamped && cx + nx <= g.dx && rows <= 2 * kQueryLanes;
    int lo[2] = {0, 0}, num[2] = {0, 0};
    if (by_rows) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int row = sub + h * kQueryLanes;
            if (row >= (int)rows) break;
            const int iz = row / ny, iy = row - iz * ny;
            const int cz = wrap_cell(zl + iz, g.dz);
            const int cy = wrap_cell(yl + iy, g.dy);
            const int2* cell = g.ranges + (cz * g.dy + cy) * g.dx + cx;
            int first = 0x7fffffff, end = 0;
#pragma unroll 3
            for (int c = 0; c < nx; ++c) {
                const int2 se = __ldg(cell + c);
                if (se.y > se.x && in_bounds(se.x >= 0 && se.y <= g.n)) {
                    first = min(first, se.x);
                    end = max(end, se.y);
                }
            }
            lo[h] = first;
            num[h] = max(end - first, 0);
        }
    }
    // candidates before row `sub`, and of all rows (rows sub + kQueryLanes follow all of the first)
    int before[2], total = 0;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        int inc = num[h];
#pragma unroll
        for (int o = 1; o < kQueryLanes; o <<= 1) {
            const int y = __shfl_up_sync(kAll, inc, o, kQueryLanes);
            if (sub >= o) inc += y;
        }
        before[h] = total + inc - num[h];
        total += __shfl_sync(kAll, inc, kQueryLanes - 1, kQueryLanes);
    }
    if (!live) return;
    if (!by_rows) {
        if (sub != 0) return;
        long long o = out ? offsets[t] : 0;
        int c = 0;
        for_each_run(g, px, py, pz, radius, [&](int l, int h) {
            c += h - l;
            if (out)
                for (int k = l; k < h; ++k) out[o++] = g.ids[k];
        });
        if (!out) counts[t] = c;
        return;
    }
    if (!out) {
        if (sub == 0) counts[t] = total;
        return;
    }
    int* o = out + offsets[t];
#pragma unroll
    for (int h = 0; h < 2; ++h)
        for (int k = 0; k < num[h]; ++k) o[before[h] + k] = __ldg(g.ids + lo[h] + k);
}

inline int ntiles_of(int n, int items = kSortItems)
{
    const int tile = kSortThreads * items;
    return (n + tile - 1) / tile;
}

// Small builds use tiles of 512 keys (2 per thread), so that a build of 65k
// points runs 128 CTAs instead of 32.
constexpr int kSmallItems = 2;
// the counting build runs on single-world grids of at most kCountMaxCells
// cells when the table has at most kCountCellsPerPoint cells per point (its
// scan reads every cell; the radix sort's cost does not grow with the table)
constexpr long long kCountMaxCells = 1LL << 26;
constexpr int kCountCellsPerPoint = 16;
constexpr int kSmallBuildPoints = 1 << 18;
inline int items_for(int n) { return n <= kSmallBuildPoints ? kSmallItems : kSortItems; }

// per-tile histogram rows the table needs for builds of up to `capacity` points
inline int hist_tiles(int capacity)
{
    return std::max(ntiles_of(capacity, kSortItems), ntiles_of(std::min(capacity, kSmallBuildPoints), kSmallItems));
}

template <int kItems>
cudaError_t load_sort_kernels()
{
    cudaFuncAttributes fa;
    cudaError_t e = cudaFuncGetAttributes(&fa, k_hash_hist<kItems>);
    if (e == cudaSuccess) e = cudaFuncGetAttributes(&fa, k_upsweep<kItems>);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_downsweep<false, kItems>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)sizeof(DownsweepSmem<kItems>));
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_downsweep<true, kItems>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)sizeof(DownsweepSmem<kItems>));
    return e;
}

}  // namespace

// --------------------------------------------------------------------------
// host side
// --------------------------------------------------------------------------
int grid_init(Grid& g, int dx, int dy, int dz, int device)
{
    if (dx <= 0 || dy <= 0 || dz <= 0) return fail(NSPH_ERR_INVALID_ARG, "grid dims must be positive");
    const long long nc = (long long)dx * dy * dz;
    if (nc > (1LL << 28)) return fail(NSPH_ERR_INVALID_ARG, "grid has more than 2^28 cells");
    g.device = device;
    g.dx = dx;
    g.dy = dy;
    g.dz = dz;
    g.ncells = nc;
    int bits = 1;
    while ((1LL << bits) < nc) ++bits;
    g.key_bits = bits;
    DeviceGuard guard(device);
    if (!guard.ok) return fail(NSPH_ERR_CUDA, "cannot select CUDA device");
    NSPH_CUDA_TRY(cudaMalloc(&g.cell_ranges, sizeof(int2) * nc));
    NSPH_CUDA_TRY(cudaMemset(g.cell_ranges, 0, sizeof(int2) * nc));
    if (nc <= kCountMaxCells) {  // the counting build's per-cell counts
        NSPH_CUDA_TRY(cudaMalloc(&g.cell_count, sizeof(int) * nc));
        NSPH_CUDA_TRY(cudaMemset(g.cell_count, 0, sizeof(int) * nc));
        const size_t tiles = (size_t)((nc + kCsTile - 1) / kCsTile);
        NSPH_CUDA_TRY(cudaMalloc(&g.tile_count, sizeof(int) * tiles));
    }
    // load every kernel now, so that a later stream capture never triggers
    // lazy module loading
    cudaFuncAttributes fa;
    NSPH_CUDA_TRY(cudaFuncGetAttributes(&fa, k_cc_count));
    NSPH_CUDA_TRY(cudaFuncGetAttributes(&fa, k_cc_tile_sums));
    NSPH_CUDA_TRY(cudaFuncGetAttributes(&fa, k_cc_scan_ranges));
    NSPH_CUDA_TRY(cudaFuncGetAttributes(&fa, k_cc_scatter));
    NSPH_CUDA_TRY(cudaFuncGetAttributes(&fa, k_cc_rank));
    NSPH_CUDA_TRY(load_sort_kernels<kSortItems>());
    NSPH_CUDA_TRY(load_sort_kernels<kSmallItems>());
    NSPH_CUDA_TRY(cudaFuncGetAttributes(&fa, k_scan_rows));
    NSPH_CUDA_TRY(cudaFuncGetAttributes(&fa, k_rank_cells));
    NSPH_CUDA_TRY(cudaFuncGetAttributes(&fa, k_rank_build));
    NSPH_CUDA_TRY(cudaFuncGetAttributes(&fa, k_ranges));
    NSPH_CUDA_TRY(cudaFuncGetAttributes(&fa, k_query));
    NSPH_CUDA_TRY(cudaDeviceSynchronize());
    return NSPH_OK;
}

int grid_init_worlds(Grid& g, const int* world_dims, int world_count, int device)
{
    if (world_count <= 0 || !world_dims) return fail(NSPH_ERR_INVALID_ARG, "world_count must be positive");
    std::vector<WorldCells> wc((size_t)world_count);
    long long off = 0;
    for (int w = 0; w < world_count; ++w) {
        const int dx = world_dims[3 * w], dy = world_dims[3 * w + 1], dz = world_dims[3 * w + 2];
        if (dx <= 0 || dy <= 0 || dz <= 0) return fail(NSPH_ERR_INVALID_ARG, "world grid dims must be positive");
        wc[w] = WorldCells{dx, dy, dz, 0.f, off};
        off += (long long)dx * dy * dz;
        if (off > (1LL << 30)) return fail(NSPH_ERR_INVALID_ARG, "the worlds' grids hold more than 2^30 cells");
    }
    g.device = device;
    g.dx = g.dy = g.dz = 0;
    g.ncells = off;
    int bits = 1;
    while ((1LL << bits) < off) ++bits;
    g.key_bits = bits;
    g.world_count = world_count;
    DeviceGuard guard(device);
    if (!guard.ok) return fail(NSPH_ERR_CUDA, "cannot select CUDA device");
    NSPH_CUDA_TRY(cudaMalloc(&g.cell_ranges, sizeof(int2) * off));
    NSPH_CUDA_TRY(cudaMemset(g.cell_ranges, 0, sizeof(int2) * off));
    NSPH_CUDA_TRY(cudaMalloc(&g.worlds, sizeof(WorldCells) * world_count));
    NSPH_CUDA_TRY(cudaMemcpy(g.worlds, wc.data(), sizeof(WorldCells) * world_count, cudaMemcpyHostToDevice));
    cudaFuncAttributes fa;
    NSPH_CUDA_TRY(load_sort_kernels<kSortItems>());
    NSPH_CUDA_TRY(load_sort_kernels<kSmallItems>());
    NSPH_CUDA_TRY(cudaFuncGetAttributes(&fa, k_scan_rows));
    NSPH_CUDA_TRY(cudaFuncGetAttributes(&fa, k_rank_cells));
    NSPH_CUDA_TRY(cudaFuncGetAttributes(&fa, k_rank_build));
    NSPH_CUDA_TRY(cudaFuncGetAttributes(&fa, k_ranges));
    NSPH_CUDA_TRY(cudaDeviceSynchronize());
    return NSPH_OK;
}

int grid_reserve(Grid& g, int capacity)
{
    if (capacity < 0) return fail(NSPH_ERR_INVALID_ARG, "negative capacity");
    if (capacity <= g.capacity) return NSPH_OK;
    DeviceGuard guard(g.device);
    if (!guard.ok) return fail(NSPH_ERR_CUDA, "cannot select CUDA device");
    // a grown reservation drops the previous build (the Warp contract)
    if (g.built && g.num_points > 0) {
        NSPH_CUDA_TRY(cudaDeviceSynchronize());
        NSPH_CUDA_TRY(cudaMemset(g.cell_ranges, 0, sizeof(int2) * g.ncells));
    }
    g.built = 0;
    g.num_points = 0;
    cudaFree(g.block);
    g.block = nullptr;
    g.keys_a = g.vals_a = g.keys_b = g.vals_b = g.point_cells = g.point_ids = nullptr;
    g.hist = g.bounds = nullptr;
    g.capacity = 0;
    // One allocation: a first build reserves on demand, and a buffer of 2^20 ints
    // and a little more takes up two megabytes more (first pass of a contact scene
    // of 1M particles, with its reserve: 2.9 ms with seven buffers of their own
    // size, 4.2 with room for the raycast's nodes in each, 1.2 as one).
    auto aligned = [](size_t bytes) { return (bytes + 255) & ~(size_t)255; };
    // a tree leaf of the raycast is 32 bytes for up to eight points
    const size_t sort = aligned(sizeof(int) * (size_t)capacity + 32);
    // per-tile digit histograms plus kRadix digit totals
    const size_t hist = aligned(sizeof(unsigned) * kRadix * ((size_t)std::max(1, hist_tiles(capacity)) + 1));
    const cudaError_t e = cudaMalloc(&g.block, 6 * sort + hist + aligned(6 * sizeof(unsigned)));
    if (e != cudaSuccess) {
        cudaGetLastError();
        g.block = nullptr;
        return fail(NSPH_ERR_OUT_OF_MEMORY, std::string("reserve: ") + cudaGetErrorString(e));
    }
    int** bufs[6] = {&g.keys_a, &g.vals_a, &g.keys_b, &g.vals_b, &g.point_cells, &g.point_ids};
    for (int b = 0; b < 6; ++b) *bufs[b] = reinterpret_cast<int*>(g.block + b * sort);
    g.hist = reinterpret_cast<unsigned*>(g.block + 6 * sort);
    g.bounds = reinterpret_cast<unsigned*>(g.block + 6 * sort + hist);
    g.capacity = capacity;
    return NSPH_OK;
}

void grid_free(Grid& g)
{
    DeviceGuard guard(g.device);
    cudaFree(g.block);
    cudaFree(g.cell_ranges);
    cudaFree(g.cell_count);
    cudaFree(g.tile_count);
    cudaFree(g.worlds);
    g = Grid();
}

namespace {

// hash, digit passes and ranges of one build with tiles of 256 x kItems keys
template <int kItems>
int build_passes(Grid& g, const float* points, int n, float cell_inv, const GatherArgs* gather, unsigned int* status,
                 cudaStream_t stream, int& nl, const int* world, int prev_n)
{
    constexpr size_t kSmem = sizeof(DownsweepSmem<kItems>);
    const int ntiles = ntiles_of(n, kItems);
    const int launch_tiles = std::max(ntiles, ntiles_of(prev_n, kItems));
    const int passes = (g.key_bits + kRadixBits - 1) / kRadixBits;
    auto mask_of = [&](int p) {
        const int bits = std::min(kRadixBits, g.key_bits - p * kRadixBits);
        return (1 << bits) - 1;
    };
    if (launch_tiles > 0) {
        NSPH_CUDA_TRY(launch_dependent(k_hash_hist<kItems>, launch_tiles, kSortThreads, 0, stream,
                                       points, n, cell_inv, g.dx, g.dy, g.dz, g.keys_a, g.vals_a, g.hist, ntiles, mask_of(0), g.point_cells, prev_n, g.cell_ranges, status, world, g.worlds, g.world_count));
        NSPH_LAUNCH_CHECK("k_hash_hist");
        ++nl;
    }
    if (n > 0) {
        const int* kin = g.keys_a;
        const int* vin = g.vals_a;
        unsigned* digit_tot = g.hist + (size_t)kRadix * hist_tiles(g.capacity);
        for (int p = 0; p < passes; ++p) {
            const bool last = (p == passes - 1);
            int* kout = last ? g.point_cells : ((p & 1) ? g.keys_a : g.keys_b);
            int* vout = last ? g.point_ids : ((p & 1) ? g.vals_a : g.vals_b);
            const int shift = p * kRadixBits;
            if (p > 0) {
                NSPH_CUDA_TRY(launch_dependent(k_upsweep<kItems>, ntiles, kSortThreads, 0, stream,
                                               kin, n, shift, mask_of(p), g.hist, ntiles));
                NSPH_LAUNCH_CHECK("k_upsweep");
                ++nl;
            }
            NSPH_CUDA_TRY(launch_dependent(k_scan_rows, kRadix, kScanThreads, 0, stream,
                                           g.hist, ntiles, digit_tot));
            NSPH_LAUNCH_CHECK("k_scan_rows");
            ++nl;
            GatherArgs ga{};
            if (last && gather) {
                ga = *gather;
                NSPH_CUDA_TRY(launch_dependent(k_downsweep<true, kItems>, ntiles, kSortThreads, kSmem, stream,
                                               kin, vin, kout, vout, n, shift, mask_of(p), g.hist, ntiles, digit_tot, ga));
            } else {
                NSPH_CUDA_TRY(launch_dependent(k_downsweep<false, kItems>, ntiles, kSortThreads, kSmem, stream,
                                               kin, vin, kout, vout, n, shift, mask_of(p), g.hist, ntiles, digit_tot, ga));
            }
            NSPH_LAUNCH_CHECK("k_downsweep");
            ++nl;
            kin = kout;
            vin = vout;
        }
        NSPH_CUDA_TRY(launch_dependent(k_ranges, (n + 255) / 256, 256, 0, stream,
                                       g.point_cells, n, g.cell_ranges));
        NSPH_LAUNCH_CHECK("k_ranges");
        ++nl;
    }
    return NSPH_OK;
}

template <int kItems>
int sort_keys(Grid& g, int n, int bits, cudaStream_t stream)
{
    const int ntiles = ntiles_of(n, kItems);
    unsigned* digit_tot = g.hist + (size_t)kRadix * hist_tiles(g.capacity);
    int *kin = g.keys_a, *vin = g.vals_a, *kout = g.keys_b, *vout = g.vals_b;
    for (int shift = 0; shift < bits; shift += kRadixBits) {
        const int mask = (1 << std::min(kRadixBits, bits - shift)) - 1;
        NSPH_CUDA_TRY(launch_dependent(k_upsweep<kItems>, ntiles, kSortThreads, 0, stream,
                                       kin, n, shift, mask, g.hist, ntiles));
        NSPH_LAUNCH_CHECK("k_upsweep");
        NSPH_CUDA_TRY(launch_dependent(k_scan_rows, kRadix, kScanThreads, 0, stream,
                                       g.hist, ntiles, digit_tot));
        NSPH_LAUNCH_CHECK("k_scan_rows");
        NSPH_CUDA_TRY(launch_dependent(k_downsweep<false, kItems>, ntiles, kSortThreads, sizeof(DownsweepSmem<kItems>), stream,
                                       kin, vin, kout, vout, n, shift, mask, g.hist, ntiles, digit_tot, GatherArgs{}));
        NSPH_LAUNCH_CHECK("k_downsweep");
        std::swap(kin, kout);
        std::swap(vin, vout);
    }
    return NSPH_OK;
}

// the counting build (see k_cc_count): 5 launches
int count_build(Grid& g, const float* points, int n, float cell_inv, const GatherArgs* gather, unsigned int* status,
                cudaStream_t stream, int& nl, int prev_n)
{
    const int tiles = (int)((g.ncells + kCsTile - 1) / kCsTile);
    // a point per thread: with four, 64k points left half of the SMs without a
    // block (count kernel 11 us; 64k rollout with its gradient 3.9 -> 3.65 ms,
    // step of 32,768 60 -> 55 us, of 1M the same)
    const int blocks = (n + 255) / 256;
    NSPH_CUDA_TRY(launch_dependent(k_cc_count, blocks, 256, 0, stream,
                                   points, n, cell_inv, g.dx, g.dy, g.dz, g.cell_count, g.keys_a, g.vals_a, g.point_cells, prev_n, g.cell_ranges, status));
    NSPH_LAUNCH_CHECK("k_cc_count");
    NSPH_CUDA_TRY(launch_dependent(k_cc_tile_sums, tiles, kCsThreads, 0, stream,
                                   g.cell_count, g.ncells, g.tile_count));
    NSPH_LAUNCH_CHECK("k_cc_tile_sums");
    NSPH_CUDA_TRY(launch_dependent(k_cc_scan_ranges, tiles, kCsThreads, 0, stream,
                                   g.cell_count, g.tile_count, g.ncells, g.cell_ranges));
    NSPH_LAUNCH_CHECK("k_cc_scan_ranges");
    NSPH_CUDA_TRY(launch_dependent(k_cc_scatter, blocks, 256, 0, stream,
                                   g.keys_a, g.vals_a, g.cell_ranges, n, g.keys_b, g.vals_b));
    NSPH_LAUNCH_CHECK("k_cc_scatter");
    NSPH_CUDA_TRY(launch_dependent(k_cc_rank, blocks, 256, 0, stream,
                                   g.vals_b, g.cell_ranges, g.keys_b, n, g.cell_count, g.point_cells, g.point_ids, gather ? *gather : GatherArgs{}, gather != nullptr));
    NSPH_LAUNCH_CHECK("k_cc_rank");
    nl += 5;
    return NSPH_OK;
}

}  // namespace

int grid_sort_keys(Grid& g, int n, int bits, cudaStream_t stream)
{
    if (n > g.capacity) return fail(NSPH_ERR_CAPACITY, "sort: more keys than reserved");
    if (n <= 0) return NSPH_OK;
    return items_for(n) == kSmallItems ? sort_keys<kSmallItems>(g, n, bits, stream)
                                       : sort_keys<kSortItems>(g, n, bits, stream);
}

int grid_build(Grid& g, const float* points, int n, float cell_width, float cell_inv, const GatherArgs* gather,
               unsigned int* status, cudaStream_t stream, int* launches, const int* world)
{
    int local_launches = 0;
    int& nl = launches ? *launches : local_launches;
    if (n < 0) return fail(NSPH_ERR_INVALID_ARG, "negative point count");
    if (n > g.capacity) return fail(NSPH_ERR_CAPACITY, "build: more points than reserved");
    if (n > 0 && !points) return fail(NSPH_ERR_INVALID_ARG, "build: null points");
    const int prev_n = g.built ? g.num_points : 0;
    const bool counting = g.world_count == 0 && g.cell_count && g.ncells <= (long long)kCountCellsPerPoint * n;
    if (n > 0 && n <= kRankMax && prev_n <= kRankPrev) {
        NSPH_CUDA_TRY(launch_dependent(k_rank_cells, (std::max(n, prev_n) + kRankThreads - 1) / kRankThreads,
                                       kRankThreads, 0, stream, points, n, cell_inv, g.dx, g.dy, g.dz, g.keys_a,
                                       g.point_cells, prev_n, g.cell_ranges, status, world, g.worlds, g.world_count));
        constexpr int kBlockPoints = kRankPoints * (kRankThreads / 32);
        NSPH_CUDA_TRY(launch_dependent(k_rank_build, (n + kBlockPoints - 1) / kBlockPoints, kRankThreads, 0, stream,
                                       g.keys_a, n, g.cell_ranges, g.point_cells, g.point_ids,
                                       gather ? *gather : GatherArgs{}, gather != nullptr));
        nl += 2;
        g.num_points = n;
        g.cell_width = cell_width;
        g.cell_inv = cell_inv;
        g.built = 1;
        return NSPH_OK;
    }
    if (counting && n > 0) {
        const int st = count_build(g, points, n, cell_inv, gather, status, stream, nl, prev_n);
        if (st != NSPH_OK) return st;
        g.num_points = n;
        g.cell_width = cell_width;
        g.cell_inv = cell_inv;
        g.built = 1;
        return NSPH_OK;
    }
    const int st = items_for(n) == kSmallItems
                       ? build_passes<kSmallItems>(g, points, n, cell_inv, gather, status, stream, nl, world, prev_n)
                       : build_passes<kSortItems>(g, points, n, cell_inv, gather, status, stream, nl, world, prev_n);
    if (st != NSPH_OK) return st;
    g.num_points = n;
    g.cell_width = cell_width;
    g.cell_inv = cell_inv;
    g.built = 1;
    return NSPH_OK;
}

}  // namespace nsph

// ==========================================================================
// C ABI: HashGrid
// ==========================================================================

using namespace nsph;

extern "C" int nsph_grid_create(int dim_x, int dim_y, int dim_z, int device, nsph_grid** out)
{
    clear_error();
    if (!out) return fail(NSPH_ERR_INVALID_ARG, "null out pointer");
    *out = nullptr;
    nsph_grid* h = new (std::nothrow) nsph_grid();
    if (!h) return fail(NSPH_ERR_OUT_OF_MEMORY, "host allocation failed");
    const int st = grid_init(h->g, dim_x, dim_y, dim_z, device);
    if (st != NSPH_OK) {
        grid_free(h->g);
        delete h;
        return st;
    }
    *out = h;
    return NSPH_OK;
}

extern "C" int nsph_grid_destroy(nsph_grid* grid)
{
    clear_error();
    if (!grid) return NSPH_OK;
    {
        DeviceGuard guard(grid->g.device);
        cudaFree(grid->mirror);
        if (grid->raycast_done) cudaEventDestroy(grid->raycast_done);
    }
    grid_free(grid->g);
    delete grid;
    return NSPH_OK;
}

extern "C" int nsph_grid_reserve(nsph_grid* grid, int num_points)
{
    clear_error();
    if (!grid) return fail(NSPH_ERR_INVALID_ARG, "null grid");
    const int st = grid_reserve(grid->g, num_points);
    if (st != NSPH_OK || grid->mirror_cap >= grid->g.capacity) return st;
    // sorted mirrors for the contact kernels (32 bytes per point)
    DeviceGuard guard(grid->g.device);
    if (!guard.ok) return fail(NSPH_ERR_CUDA, "cannot select CUDA device");
    cudaFree(grid->mirror);
    grid->mirror = nullptr;
    grid->mirror_cap = 0;
    const size_t c = (size_t)std::max(1, grid->g.capacity);
    if (cudaMalloc(&grid->mirror, sizeof(float4) * 2 * c) != cudaSuccess) {
        cudaGetLastError();
        grid->mirror = nullptr;
        return fail(NSPH_ERR_OUT_OF_MEMORY, "grid reserve: contact mirror allocation failed");
    }
    grid->mirror_cap = grid->g.capacity;
    return NSPH_OK;
}

extern "C" int nsph_grid_build(nsph_grid* grid, const float* points, int num_points, float radius, void* stream)
{
    clear_error();
    NvtxRange nvtx_range("nsph_grid_build");
    if (!grid) return fail(NSPH_ERR_INVALID_ARG, "null grid");
    if (!(radius > 0.f) || !isfinite(radius)) return fail(NSPH_ERR_INVALID_ARG, "radius must be positive and finite");
    DeviceGuard guard(grid->g.device);
    if (!guard.ok) return fail(NSPH_ERR_CUDA, "cannot select CUDA device");
    const float inv = 1.0f / radius;
    int launches = 0;
    const int st = grid_build(grid->g, points, num_points, radius, inv, nullptr, nullptr, (cudaStream_t)stream,
                              &launches);
    grid->g.last_launches = launches;
    return st;
}

extern "C" int nsph_grid_last_launches(const nsph_grid* grid) { return grid ? grid->g.last_launches : 0; }

extern "C" int nsph_grid_get_view(const nsph_grid* grid, nsph_grid_view* view)
{
    clear_error();
    if (!grid || !view) return fail(NSPH_ERR_INVALID_ARG, "null argument");
    const Grid& g = grid->g;
    view->point_cells = g.point_cells;
    view->point_ids = g.point_ids;
    view->cell_starts = reinterpret_cast<const int*>(g.cell_ranges);
    view->cell_ends = reinterpret_cast<const int*>(g.cell_ranges) + 1;
    view->cell_stride = 2;
    view->num_points = g.num_points;
    view->dim_x = g.dx;
    view->dim_y = g.dy;
    view->dim_z = g.dz;
    view->cell_width = g.cell_width;
    view->cell_width_inv = g.cell_inv;
    view->built = g.built;
    return NSPH_OK;
}

extern "C" int nsph_grid_query(const nsph_grid* grid, const float* queries, int num_queries, float radius,
                               int* counts, const long long* offsets, int* out_ids, void* stream)
{
    clear_error();
    NvtxRange nvtx_range("nsph_grid_query");
    if (!grid) return fail(NSPH_ERR_INVALID_ARG, "null grid");
    if (!grid->g.built) return fail(NSPH_ERR_NOT_BUILT, "query before build");
    if (num_queries < 0) return fail(NSPH_ERR_INVALID_ARG, "negative query count");
    if (num_queries == 0) return NSPH_OK;
    if (!queries) return fail(NSPH_ERR_INVALID_ARG, "null queries");
    if (out_ids ? !offsets : !counts) return fail(NSPH_ERR_INVALID_ARG, "counts (count call) or offsets (fill call) required");
    DeviceGuard guard(grid->g.device);
    if (!guard.ok) return fail(NSPH_ERR_CUDA, "cannot select CUDA device");
    NSPH_CUDA_TRY(launch_dependent(k_query, (unsigned)(((long long)num_queries * kQueryLanes + 127) / 128), 128, 0, (cudaStream_t)stream,
                                   grid->g.view(), queries, num_queries, radius, counts, offsets, out_ids));
    NSPH_LAUNCH_CHECK("k_query");
    return NSPH_OK;
}

// ==========================================================================
// C ABI: allocation-free HashGrid build
//
// For callers that must not allocate device memory: code that rebuilds the
// grid while a CUDA stream is being captured (cudaMalloc is not allowed
// during a global-mode capture), and host programs whose device memory is
// owned by another allocator (a framework's caching allocator or a fixed
// arena, where a library-side cudaMalloc would compete for memory and
// synchronise the device). The caller passes the points and every output;
// the sort scratch lives in the fixed device array below.
// ==========================================================================
namespace nsph {
namespace {

// Every accepted size is a small build, so the sort uses the small builds'
// 512-key tiles, like nsph_grid_build does for the same point count.
static_assert(NSPH_NOALLOC_MAX_POINTS <= kSmallBuildPoints, "allocation-free builds are small builds");
constexpr int kNoAllocItems = kSmallItems;
constexpr int kNoAllocTiles = (NSPH_NOALLOC_MAX_POINTS + kSortThreads * kNoAllocItems - 1) /
                              (kSortThreads * kNoAllocItems);
// keys_a, vals_a, keys_b, vals_b (NSPH_NOALLOC_MAX_POINTS ints each), then
// the per-tile digit histograms and the kRadix digit totals
constexpr size_t kNoAllocSortInts = 4 * (size_t)NSPH_NOALLOC_MAX_POINTS;
constexpr size_t kNoAllocHistUints = (size_t)kRadix * (kNoAllocTiles + 1);
constexpr size_t kNoAllocBytes = sizeof(int) * kNoAllocSortInts + sizeof(unsigned) * kNoAllocHistUints;

// Held by every GPU that loads the library until the process exits. Shared by
// all calls: the last call's contents stay behind, and calls that overlap on
// the GPU race on it.
static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocBytes];

// start / end of each cell into two caller arrays (Warp's layout)
__global__ void k_ranges_split(const int* __restrict__ cells, int n, int* __restrict__ starts, int* __restrict__ ends)
{
    launch_entry();
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const int c = cells[k];
    if (k == 0 || cells[k - 1] != c) starts[c] = k;
    if (k == n - 1 || cells[k + 1] != c) ends[c] = k + 1;
}

constexpr int kNoAllocMaxDevices = 64;
unsigned char* g_noalloc_ptr[kNoAllocMaxDevices] = {};  // device address per device
std::mutex g_noalloc_mutex;

// Device address of g_noalloc_scratch on the current device (looked up once
// per device with that device current; in host code the symbol itself is only
// a host-side stand-in and must never be handed to a kernel).
int noalloc_scratch(int device, unsigned char** out)
{
    if (device < 0 || device >= kNoAllocMaxDevices) return fail(NSPH_ERR_INVALID_ARG, "device ordinal out of range");
    std::lock_guard<std::mutex> lock(g_noalloc_mutex);
    if (!g_noalloc_ptr[device]) {
        void* ptr = nullptr;
        NSPH_CUDA_TRY(cudaGetSymbolAddress(&ptr, g_noalloc_scratch));
        // load every kernel a build may launch now, so that no later call
        // (whatever its size, even the first one inside a stream capture)
        // triggers lazy module loading
        cudaFuncAttributes fa;
        NSPH_CUDA_TRY(load_sort_kernels<kNoAllocItems>());
        NSPH_CUDA_TRY(cudaFuncGetAttributes(&fa, k_scan_rows));
        NSPH_CUDA_TRY(cudaFuncGetAttributes(&fa, k_ranges_split));
        g_noalloc_ptr[device] = static_cast<unsigned char*>(ptr);
    }
    *out = g_noalloc_ptr[device];
    return NSPH_OK;
}

}  // namespace
}  // namespace nsph

extern "C" int nsph_grid_build_noalloc(const float* points, int num_points, float radius, int dim_x, int dim_y,
                                       int dim_z, int* point_cells, int* point_ids, int* cell_starts, int* cell_ends,
                                       void* stream)
{
    clear_error();
    NvtxRange nvtx_range("nsph_grid_build_noalloc");
    if (num_points < 0) return fail(NSPH_ERR_INVALID_ARG, "negative point count");
    if (num_points > NSPH_NOALLOC_MAX_POINTS)
        return fail(NSPH_ERR_CAPACITY, "nsph_grid_build_noalloc: more than NSPH_NOALLOC_MAX_POINTS (" +
                                           std::to_string(NSPH_NOALLOC_MAX_POINTS) + ") points");
    if (dim_x <= 0 || dim_y <= 0 || dim_z <= 0) return fail(NSPH_ERR_INVALID_ARG, "grid dims must be positive");
    const long long ncells = (long long)dim_x * dim_y * dim_z;
    if (ncells > (1LL << 28)) return fail(NSPH_ERR_INVALID_ARG, "grid has more than 2^28 cells");
    if (!(radius > 0.f) || !isfinite(radius)) return fail(NSPH_ERR_INVALID_ARG, "radius must be positive and finite");
    if (!cell_starts || !cell_ends || (num_points > 0 && (!points || !point_cells || !point_ids)))
        return fail(NSPH_ERR_INVALID_ARG, "null pointer");
    int device = 0;
    NSPH_CUDA_TRY(cudaGetDevice(&device));
    unsigned char* scratch = nullptr;
    int st = noalloc_scratch(device, &scratch);
    if (st != NSPH_OK) return st;
    cudaStream_t cs = (cudaStream_t)stream;
    int* keys_a = reinterpret_cast<int*>(scratch);
    int* vals_a = keys_a + NSPH_NOALLOC_MAX_POINTS;
    int* keys_b = vals_a + NSPH_NOALLOC_MAX_POINTS;
    int* vals_b = keys_b + NSPH_NOALLOC_MAX_POINTS;
    unsigned* hist = reinterpret_cast<unsigned*>(vals_b + NSPH_NOALLOC_MAX_POINTS);
    unsigned* digit_tot = hist + (size_t)kRadix * kNoAllocTiles;
    // empty cells read 0/0
    NSPH_CUDA_TRY(cudaMemsetAsync(cell_starts, 0, sizeof(int) * ncells, cs));
    NSPH_CUDA_TRY(cudaMemsetAsync(cell_ends, 0, sizeof(int) * ncells, cs));
    const int n = num_points;
    if (n == 0) return NSPH_OK;
    int bits = 1;
    while ((1LL << bits) < ncells) ++bits;
    const int passes = (bits + kRadixBits - 1) / kRadixBits;
    auto mask_of = [&](int p) { return (1 << std::min(kRadixBits, bits - p * kRadixBits)) - 1; };
    const int ntiles = ntiles_of(n, kNoAllocItems);
    const float inv = 1.0f / radius;
    NSPH_CUDA_TRY(launch_dependent(k_hash_hist<kNoAllocItems>, ntiles, kSortThreads, 0, cs,
                                   points, n, inv, dim_x, dim_y, dim_z, keys_a, vals_a, hist, ntiles, mask_of(0), nullptr, 0, nullptr, nullptr, nullptr, nullptr, 0));
    NSPH_LAUNCH_CHECK("k_hash_hist");
    const int* kin = keys_a;
    const int* vin = vals_a;
    for (int p = 0; p < passes; ++p) {
        const bool last = (p == passes - 1);
        int* kout = last ? point_cells : ((p & 1) ? keys_a : keys_b);
        int* vout = last ? point_ids : ((p & 1) ? vals_a : vals_b);
        const int shift = p * kRadixBits;
        if (p > 0) {
            NSPH_CUDA_TRY(launch_dependent(k_upsweep<kNoAllocItems>, ntiles, kSortThreads, 0, cs,
                                           kin, n, shift, mask_of(p), hist, ntiles));
            NSPH_LAUNCH_CHECK("k_upsweep");
        }
        NSPH_CUDA_TRY(launch_dependent(k_scan_rows, kRadix, kScanThreads, 0, cs,
                                       hist, ntiles, digit_tot));
        NSPH_LAUNCH_CHECK("k_scan_rows");
        NSPH_CUDA_TRY(launch_dependent(k_downsweep<false, kNoAllocItems>, ntiles, kSortThreads, sizeof(DownsweepSmem<kNoAllocItems>), cs,
                                       kin, vin, kout, vout, n, shift, mask_of(p), hist, ntiles, digit_tot, GatherArgs{}));
        NSPH_LAUNCH_CHECK("k_downsweep");
        kin = kout;
        vin = vout;
    }
    NSPH_CUDA_TRY(launch_dependent(k_ranges_split, (n + 255) / 256, 256, 0, cs,
                                   point_cells, n, cell_starts, cell_ends));
    NSPH_LAUNCH_CHECK("k_ranges_split");
    return NSPH_OK;
}
