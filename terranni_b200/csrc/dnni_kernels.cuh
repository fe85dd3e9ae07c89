// dnni_kernels.cuh -- sm_100a kernels of the discrete natural-neighbour
// interpolation hot path, for a batch of work packages ("tiles") at once.
//
// Replaces, per work package:
//   nni.cpp:722-790 renderInputPoints / nni.cpp:171-230 drawPlane (the GL
//     depth-tested site planes that leave each pixel's nearest site in the
//     colour buffer)                       -> k_region_* + k_near_dense/far
//   nni.cpp:794-820 performNNIQueries / nni.cpp:483-534 makeBlocks and
//     cuda_nni.cu:407-488 calcNNI (query planes OR-blended into bit masks,
//     then per-pixel int32 atomics)        -> k_scatter_window + k_rows_final stencil
//   cuda_nni.cu:491-503 divide, cuda_nni.cu:399-402 zeroValues
//                                          -> k_rows_final
//
// Every kernel covers all tiles of a batch in one launch: its blocks (or
// warps, or threads) are numbered across the tiles and an exclusive prefix
// array per kind of work (point chunks, scan blocks, raster tiles, ...) maps
// a block back to its tile.  A single work package is a batch of one.
// Nothing here waits on the host, so a batch's whole launch sequence can be
// captured in one CUDA graph.
//
// Data layout in HBM (per tile, at the offsets in TileParams):
//   sorted points  int4 {x-ox, y-oy, z, gid}, grouped by search bin;
//   bin starts     int32 [nbins+1], bins ordered superblock (64x64 bins) ->
//                  block (8x8 bins) -> bin, so any bin, block or superblock is
//                  one contiguous point range;
//   occupancy      one 64-bit mask per block (its bins) and per superblock
//                  (its blocks); a nearest non-empty block per block;
//   pixel records  int2 {z of nearest site, R2 = floor(d^2/cell^2)} per
//                  raster pixel (R2 = -1: no site);
//   span words     one 64-bit word per grid cell holding (Zrel << K) + C, or
//                  int64 Z plus int32 C when the packed form cannot hold the
//                  largest possible per-cell sums.
#pragma once

#include <cuda_pipeline_primitives.h>

#include "dnni_search.cuh"

namespace dnni {

constexpr int kChunkLarge = 4096, kChunkSmall = 2048;   // points per block in the point passes (BatchTables::chunk)
constexpr int kChunkThreads = 512;
constexpr int kScanThreads = 256;
constexpr int kScanItems = 16;
constexpr int kScanTile = kScanThreads * kScanItems;   // counts per scan block

// Prefix arrays of one batch (each of length ntiles + 1, first entry 0).
struct BatchTables {
    const TileParams* tiles;
    int ntiles;
    int chunk;                   // points per block in the point passes
    const int* chunk_base;       // point chunks
    const int* scan_base;        // scan blocks of kScanTile counts (and block-sum slots)
    const int64_t* blk_base;     // blocks (== TileParams::blk_off)
    const int64_t* sup_base;     // superblocks (== TileParams::sup_off)
    const int* row1_base;        // rows of the block grid
    const int* rt_base;          // 32 x kTileY raster tiles
    const int* ct_base;          // 32 x 16 cell tiles
    const int* grow_base;        // grid rows
    const int* band_base;        // bands of 16 grid rows
    const int* strip_base;       // binning regions of 512 bins
    const int* whole_base;       // and of 4096 bins
};

struct BatchCounters {
    int nfar;                    // far groups listed
    int err;                     // kErrRange when a point was out of range
    int far_next;                // next far group to hand out
    int nspan;                   // span work items listed
    int span_next;               // next span work item to hand out
    int nheavy;                  // far groups left to the heavy pass
    int heavy_next;              // next of them to hand out
    int ticket;                  // blocks of the bounding-box pass, then of the heavy pass, that have finished
};

// First statement of the kernels that a single work package's call launches as a
// chain: waits until the kernel before has finished and its writes are visible,
// then lets the next one's blocks be placed while this one runs (they wait here
// in turn).  Without the launch attribute both do nothing.
__device__ __forceinline__ void chained() {
    cudaGridDependencySynchronize();
    cudaTriggerProgrammaticLaunchCompletion();
}

template <typename B>
__device__ __forceinline__ int find_tile(const B* __restrict__ base, int ntiles, long long k) {
    int lo = 0, hi = ntiles - 1;   // last tile with base[t] <= k
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if ((long long)__ldg(&base[mid]) <= k) lo = mid; else hi = mid - 1;
    }
    return lo;
}

// ---------------------------------------------------------------------------
// point passes
// ---------------------------------------------------------------------------

// The region arrays live in the tile's part of the bin-count array: counts,
// then starts (regions + 1), then cursors; 3 (nbins >> rsh) + 1 <= nbins.
struct RegionArrays {
    int *cnt, *start, *cur;
};
__device__ __forceinline__ RegionArrays region_arrays(const TileParams& T, int* bins) {
    const int n = (int)(T.bg.nbins >> T.rsh);
    RegionArrays r;
    r.cnt = bins + T.bin_off;
    r.start = r.cnt + n;
    r.cur = r.start + n + 1;
    return r;
}

// rtmax (optional): the raster tiles' largest R2; bins (optional): the tiles'
// region counts, which start at zero.
__global__ void __launch_bounds__(256) k_init_scalars(BatchTables bt, Scalars* sc, BatchCounters* ctr, int* rtmax,
                                                      int* bins) {
    const int t = blockIdx.x, l = threadIdx.x;
    Scalars* s = sc + t;
    if (rtmax)
        for (int k = bt.rt_base[t] + l; k < bt.rt_base[t + 1]; k += blockDim.x) rtmax[k] = -1;
    if (bins) {
        const RegionArrays r = region_arrays(bt.tiles[t], bins);
        for (int k = l; k < (int)(bt.tiles[t].bg.nbins >> bt.tiles[t].rsh); k += blockDim.x) r.cnt[k] = 0;
    }
    if (l == 0) {
        s->bbox[0] = INT_MAX; s->bbox[1] = INT_MIN;
        s->bbox[2] = INT_MAX; s->bbox[3] = INT_MIN;
        s->bbox[4] = INT_MAX; s->bbox[5] = INT_MIN;
        s->err = 0; s->packed = 0; s->kbits = 0; s->ticket = 0; s->zbase = 0;
        if (t == 0) { ctr->nfar = 0; ctr->err = 0; ctr->far_next = 0; ctr->nspan = 0; ctr->span_next = 0; ctr->nheavy = 0; ctr->heavy_next = 0; ctr->ticket = 0; }
    }
    if (l < kStatSlots) {
        s->max_r2[l] = -1; s->big_pixels[l] = 0; s->spans[l] = 0; s->nodata[l] = 0;
        s->evals_dense[l] = 0; s->evals_far[l] = 0;
    }
    if (l < kSpanHistBuckets) s->span_hist[l] = 0;
}

// A single work package's tables, passed by value: no staging buffer, copy or
// wait between the host's plan and the kernels that read it.
struct OneTable {
    uint4 w[32];
};

__device__ __forceinline__ bool last_block(int* ticket, int blocks) {
    __shared__ int last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(ticket, 1) == blocks - 1;
    __syncthreads();
    return last != 0;
}

// Writes the tables; scalars: and starts the scalars and counters, as
// k_init_scalars does; nreg: and starts that many region counts at zero.
__global__ void __launch_bounds__(256) k_init_one(OneTable tab, uint4* __restrict__ tables, int words, int scalars, Scalars* s,
                                                  BatchCounters* ctr, int* __restrict__ cnt, int nreg) {
    chained();
    const int l = threadIdx.x;
    if (blockIdx.x == 0) {
        if (l < words) tables[l] = tab.w[l];
        if (scalars) {
            for (int k = l; k < (int)(sizeof(Scalars) / sizeof(int)); k += blockDim.x) ((int*)s)[k] = 0;
            if (l < (int)(sizeof(BatchCounters) / sizeof(int))) ((int*)ctr)[l] = 0;
            __syncthreads();
            if (l < kStatSlots) s->max_r2[l] = -1;
            if (l < 6) s->bbox[l] = l & 1 ? INT_MIN : INT_MAX;
        }
    }
    for (int k = blockIdx.x * blockDim.x + l; k < nreg; k += gridDim.x * blockDim.x) cnt[k] = 0;
}

// Bounding box of each tile's points relative to its origin, with range checks
// (the coordinate range, and the declared extent where the caller gave one):
// bbox_point per point on the input coordinates, bbox_flush once per block; a
// point is out of range exactly when the block's box is.
struct BBoxAcc {
    int mnx = INT_MAX, mxx = INT_MIN, mny = INT_MAX, mxy = INT_MIN, mnz = INT_MAX, mxz = INT_MIN;
};

__device__ __forceinline__ void bbox_point(int x, int y, int z, BBoxAcc& acc) {
    acc.mnx = min(acc.mnx, x); acc.mxx = max(acc.mxx, x);
    acc.mny = min(acc.mny, y); acc.mxy = max(acc.mxy, y);
    acc.mnz = min(acc.mnz, z); acc.mxz = max(acc.mxz, z);
}

// One reduction per block (kChunkThreads threads), so that a tile's blocks
// meet in its six words once each: with one per warp the same-address atomics
// took 0.34 ms of the 0.38 ms pass over 20 M points.
__device__ __forceinline__ void bbox_flush(const TileParams& T, const BBoxAcc& acc, Scalars* s, BatchCounters* ctr) {
    __shared__ int red[6][kChunkThreads / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int v[6] = {acc.mnx, acc.mxx, acc.mny, acc.mxy, acc.mnz, acc.mxz};
#pragma unroll
    for (int k = 0; k < 6; ++k) {
        const int r = k & 1 ? __reduce_max_sync(0xffffffffu, v[k]) : __reduce_min_sync(0xffffffffu, v[k]);
        if (lane == 0) red[k][warp] = r;
    }
    __syncthreads();
    if (warp < 6) {
        // warp 0..5: least and greatest x, y, z of the block
        const bool top = warp & 1;
        const int x = red[warp][lane & (kChunkThreads / 32 - 1)];
        const int r = top ? __reduce_max_sync(0xffffffffu, x) : __reduce_min_sync(0xffffffffu, x);
        if (lane == 0) {
            const long long o = warp < 2 ? T.ox : (warp < 4 ? T.oy : 0), rel = (long long)r - o;
            bool bad = top ? rel >= kCoordLimit : rel <= -kCoordLimit;
            if (T.has_ext && warp < 4) {
                const int e = warp < 2 ? (top ? T.ex1 : T.ex0) : (top ? T.ey1 : T.ey0);
                bad |= top ? rel > e : rel < e;
            }
            if (bad) { atomicOr(&s->err, kErrRange); atomicOr(&ctr->err, kErrRange); }
            const int c = (int)min(max(rel, -kCoordLimit), kCoordLimit);
            if (top) atomicMax(&s->bbox[warp], c); else atomicMin(&s->bbox[warp], c);
        }
    }
}

// host (optional, one tile): where the last block to finish leaves the box and
// the error bits for the host, in its mapped memory.
__global__ void __launch_bounds__(kChunkThreads) k_bbox(BatchTables bt, const int32_t* __restrict__ xyz, Scalars* sc,
                                                        BatchCounters* ctr, Scalars* host) {
    chained();
    const int t = find_tile(bt.chunk_base, bt.ntiles, blockIdx.x);
    const TileParams& T = bt.tiles[t];
    const int64_t c0 = (int64_t)(blockIdx.x - __ldg(&bt.chunk_base[t])) * bt.chunk;
    const int64_t c1 = c0 + bt.chunk < T.npts ? c0 + bt.chunk : T.npts;
    const int32_t* p = xyz + 3 * T.pt_off;
    BBoxAcc acc;
    constexpr int kB = 4;                // points in flight
    for (int64_t b = c0; b < c1; b += kB * kChunkThreads) {
        int x[kB], y[kB], z[kB];
#pragma unroll
        for (int k = 0; k < kB; ++k) {
            const int64_t i = b + k * kChunkThreads + threadIdx.x;
            if (i < c1) {
                x[k] = p[3 * i];
                y[k] = p[3 * i + 1];
                z[k] = p[3 * i + 2];
            }
        }
#pragma unroll
        for (int k = 0; k < kB; ++k)
            if (b + k * kChunkThreads + threadIdx.x < c1) bbox_point(x[k], y[k], z[k], acc);
    }
    bbox_flush(T, acc, sc + t, ctr);
    if (host && last_block(&ctr->ticket, gridDim.x)) {
        if (threadIdx.x < 6) host->bbox[threadIdx.x] = __ldcg(&sc->bbox[threadIdx.x]);
        if (threadIdx.x == 6) host->err = __ldcg(&sc->err);
        if (threadIdx.x == 7) ctr->ticket = 0;
        __threadfence_system();
    }
}

// A tile's points outside its bin grid (possible only when the caller's
// declared point extent was wrong) are counted as a range error and binned
// at the grid's edge, so that no access leaves the tile's arrays.
__device__ __forceinline__ int64_t point_bin_checked(const BinGrid& g, int xr, int yr, unsigned& bad) {
    const long long ux = (long long)xr - g.gx0, uy = (long long)yr - g.gy0;
    if (ux < 0 || uy < 0 || ux >= (long long)g.nbx * g.bs || uy >= (long long)g.nby * g.bs) bad = 1;
    int bx = ux < 0 ? 0 : (ux >= (1LL << 32) ? g.nbx - 1 : udiv32(ux, g.bs));
    int by = uy < 0 ? 0 : (uy >= (1LL << 32) ? g.nby - 1 : udiv32(uy, g.bs));
    bx = bx < g.nbx - 1 ? bx : g.nbx - 1;
    by = by < g.nby - 1 ? by : g.nby - 1;
    return bin_id(g, bx, by);
}

// ---- binning by regions ----
//
// A region is a run of 2^rsh bins (a superblock or an eighth of one: a strip of
// 64 x 8 bins), so its points are one range of the sorted array.  k_region_count
// counts the points per region and turns the counts into ranges, k_region_part groups the points by region (into a part of the scratch that
// later phases use: the span words, pixel records and worklist), and
// k_region_sort sorts one region's points by bin with the counters in shared
// memory, writing the bin starts and the occupancy masks on the way.  A tile of
// one region goes straight from its input rows to k_region_sort.
//
// Bound by latency around the scattered 16-byte stores of the partition and
// the sort, then by DRAM (2.9 TB/s in the sort of 20 M points, whose superblocks
// are read twice).  Box and binning of 20 M points on 4096^2 cells 1.49 -> 0.69
// ms, of 200 mixed tiles (37.5 M points) 1.68 -> 1.07 ms against one counting
// pass with global reductions, three scan passes, one scatter with a returning
// global atomic per point and two mask passes.

// A point's bin coordinates, clamped to the grid; bad is set for a point
// outside it (possible only when the caller's declared point extent was
// wrong), which is then a range error, binned at the edge so that no access
// leaves the tile's arrays.
__device__ __forceinline__ int64_t point_bin_est(const BinGrid& g, float inv_bs, int xr, int yr, unsigned& bad) {
    const long long ux = (long long)xr - g.gx0, uy = (long long)yr - g.gy0;
    if (ux < 0 || uy < 0 || ux >= (long long)g.nbx * g.bs || uy >= (long long)g.nby * g.bs) {
        bad = 1;
        int bx = ux < 0 ? 0 : (ux >= (1LL << 32) ? g.nbx - 1 : udiv32(ux, g.bs));
        int by = uy < 0 ? 0 : (uy >= (1LL << 32) ? g.nby - 1 : udiv32(uy, g.bs));
        bx = bx < g.nbx - 1 ? bx : g.nbx - 1;
        by = by < g.nby - 1 ? by : g.nby - 1;
        return bin_id(g, bx, by);
    }
    return bin_id(g, floor_div_u32((unsigned)ux, (unsigned)g.bs, inv_bs), floor_div_u32((unsigned)uy, (unsigned)g.bs, inv_bs));
}

// with_bbox: also the bounding box and range checks of k_bbox (batches, whose
// bin grids are planned before any point is seen, skip k_bbox).
__global__ void __launch_bounds__(kChunkThreads) k_region_count(BatchTables bt, const int32_t* __restrict__ xyz,
                                                                int* __restrict__ bins, Scalars* sc, BatchCounters* ctr,
                                                                int with_bbox) {
    chained();
    extern __shared__ int hist[];
    const int t = find_tile(bt.chunk_base, bt.ntiles, blockIdx.x);
    const TileParams& T = bt.tiles[t];
    const BinGrid g = T.bg;
    const int rsh = T.rsh, nreg = (int)(g.nbins >> rsh);
    if (nreg == 1 && !with_bbox) return;
    const float inv_bs = 1.0f / (float)g.bs;
    const int64_t c0 = (int64_t)(blockIdx.x - __ldg(&bt.chunk_base[t])) * bt.chunk;
    const int64_t c1 = c0 + bt.chunk < T.npts ? c0 + bt.chunk : T.npts;
    const int32_t* p = xyz + 3 * T.pt_off;
    for (int k = threadIdx.x; k < nreg; k += kChunkThreads) hist[k] = 0;
    __syncthreads();
    unsigned bad = 0;
    BBoxAcc acc;
    constexpr int kB = 4;                // loads in flight before the first atomic
    for (int64_t b = c0; b < c1; b += kB * kChunkThreads) {
        int x[kB], y[kB], z[kB];
#pragma unroll
        for (int k = 0; k < kB; ++k) {
            const int64_t i = b + k * kChunkThreads + threadIdx.x;
            if (i < c1) {
                x[k] = p[3 * i];
                y[k] = p[3 * i + 1];
                z[k] = with_bbox ? p[3 * i + 2] : 0;
            }
        }
#pragma unroll
        for (int k = 0; k < kB; ++k) {
            if (b + k * kChunkThreads + threadIdx.x >= c1) continue;
            if (with_bbox) bbox_point(x[k], y[k], z[k], acc);
            const int64_t id = point_bin_est(g, inv_bs, rel_coord(x[k], T.ox), rel_coord(y[k], T.oy), bad);
            if (nreg > 1) atomicAdd(&hist[id >> rsh], 1);
        }
    }
    if (with_bbox) bbox_flush(T, acc, sc + t, ctr);
    if (__any_sync(0xffffffffu, bad) && (threadIdx.x & 31) == 0) atomicOr(&ctr->err, kErrRange);
    if (nreg == 1) return;
    __syncthreads();
    const RegionArrays r = region_arrays(T, bins);
    for (int k = threadIdx.x; k < nreg; k += kChunkThreads)
        if (hist[k]) atomicAdd(&r.cnt[k], hist[k]);
    // the tile's last block turns the counts into the regions' ranges
    const int blocks = __ldg(&bt.chunk_base[t + 1]) - __ldg(&bt.chunk_base[t]);
    if (!last_block(&sc[t].ticket, blocks)) return;
    __shared__ int wsum[kChunkThreads / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int carry = 0;
    for (int b = 0; b < nreg; b += 2 * kChunkThreads) {
        const int k = b + 2 * threadIdx.x;
        const int v0 = k < nreg ? __ldcg(&r.cnt[k]) : 0, v1 = k + 1 < nreg ? __ldcg(&r.cnt[k + 1]) : 0;
        int x = v0 + v1;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) { const int y = __shfl_up_sync(0xffffffffu, x, o); if (lane >= o) x += y; }
        if (lane == 31) wsum[warp] = x;
        __syncthreads();
        int w = lane < kChunkThreads / 32 ? wsum[lane] : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) { const int y = __shfl_up_sync(0xffffffffu, w, o); if (lane >= o) w += y; }
        const int before = __shfl_sync(0xffffffffu, w, (warp + 31) & 31), total = __shfl_sync(0xffffffffu, w, 31);
        const int run = carry + (warp ? before : 0) + x - v0 - v1;
        if (k < nreg) { r.start[k] = run; r.cur[k] = run; }
        if (k + 1 < nreg) { r.start[k + 1] = run + v0; r.cur[k + 1] = run + v0; }
        carry += total;
        __syncthreads();
    }
    if (threadIdx.x == 0) r.start[nreg] = carry;
}

// A chunk's points to their regions: ranks from a shared-memory histogram, one
// global reservation per region the chunk touches.
__global__ void __launch_bounds__(kChunkThreads, 2) k_region_part(BatchTables bt, const int32_t* __restrict__ xyz,
                                                               const uint32_t* __restrict__ gid, int* __restrict__ bins,
                                                               int4* __restrict__ part) {
    chained();
    extern __shared__ int hist[];
    constexpr int kPer = kChunkLarge / kChunkThreads;
    const int t = find_tile(bt.chunk_base, bt.ntiles, blockIdx.x);
    const TileParams& T = bt.tiles[t];
    const BinGrid g = T.bg;
    const int rsh = T.rsh, nreg = (int)(g.nbins >> rsh);
    if (nreg == 1) return;
    const float inv_bs = 1.0f / (float)g.bs;
    const int64_t c0 = (int64_t)(blockIdx.x - __ldg(&bt.chunk_base[t])) * bt.chunk;
    const int64_t c1 = c0 + bt.chunk < T.npts ? c0 + bt.chunk : T.npts;
    const int32_t* p = xyz + 3 * T.pt_off;
    for (int k = threadIdx.x; k < nreg; k += kChunkThreads) hist[k] = 0;
    __syncthreads();
    int x[kPer], y[kPer], z[kPer];
    unsigned at[kPer];                   // a point's region << 13 | its rank there (below kChunkLarge)
    unsigned bad = 0;
#pragma unroll
    for (int k = 0; k < kPer; ++k) {
        const int64_t i = c0 + k * kChunkThreads + threadIdx.x;
        if (i < c1) {
            x[k] = rel_coord(p[3 * i], T.ox);
            y[k] = rel_coord(p[3 * i + 1], T.oy);
            z[k] = p[3 * i + 2];
        }
    }
#pragma unroll
    for (int k = 0; k < kPer; ++k) {
        if (c0 + k * kChunkThreads + threadIdx.x >= c1) continue;
        const unsigned r = (unsigned)(point_bin_est(g, inv_bs, x[k], y[k], bad) >> rsh);
        at[k] = (r << 13) | (unsigned)atomicAdd(&hist[r], 1);
    }
    __syncthreads();
    int* cur = region_arrays(T, bins).cur;
    for (int k = threadIdx.x; k < nreg; k += kChunkThreads) {
        const int n = hist[k];
        if (n) hist[k] = atomicAdd(&cur[k], n);
    }
    __syncthreads();
    int4* out = part + T.srt_off;
#pragma unroll
    for (int k = 0; k < kPer; ++k) {
        const int64_t i = c0 + k * kChunkThreads + threadIdx.x;
        if (i < c1)
            out[hist[at[k] >> 13] + (int)(at[k] & 8191u)] = make_int4(x[k], y[k], z[k], (int)(gid ? gid[T.pt_off + i] : (uint32_t)i));
    }
}

// One region: counts its points per bin, scans, writes the bins' starts and
// occupancy masks, and places the points.  Up to kHold points per thread keep
// their bins and ranks in registers; the points themselves are read twice.  The
// order of the points inside a bin is arbitrary, which no result depends on:
// every comparison of sites orders them by (distance, gid, z), never by
// position.
//
// A strip goes to 256 threads (six CTAs per SM), its points' ranks held; a
// superblock or a tile's only region, several times larger and fewer, to 1024.
template <int kRsh>
__global__ void __launch_bounds__(kRsh == 9 ? 256 : 1024, kRsh == 9 ? 6 : 2) k_region_sort(BatchTables bt, const int32_t* __restrict__ xyz,
                                                              const uint32_t* __restrict__ gid, int* __restrict__ bins,
                                                              const int4* __restrict__ part, int* __restrict__ start_all,
                                                              int4* __restrict__ sorted, uint64_t* __restrict__ bmask,
                                                              uint64_t* __restrict__ smask) {
    chained();
    constexpr int kSortThreads = kRsh == 9 ? 256 : 1024, nb = 1 << kRsh, mask = nb - 1;
    constexpr int kHold = kRsh == 9 ? 8 : 0, kB = 4;     // kB: loads in flight before the first atomic
    __shared__ int cnt[nb + 1];
    __shared__ int wsum[kSortThreads / 32];
    __shared__ unsigned any[2];
    const int* base = kRsh == 9 ? bt.strip_base : bt.whole_base;
    const int t = find_tile(base, bt.ntiles, blockIdx.x);
    const TileParams& T = bt.tiles[t];
    const BinGrid g = T.bg;
    const int r = blockIdx.x - __ldg(&base[t]), nreg = (int)(g.nbins >> kRsh);
    const bool direct = nreg == 1;
    const RegionArrays ra = region_arrays(T, bins);
    const int s0 = direct ? 0 : ra.start[r], n = direct ? (int)T.npts : ra.start[r + 1] - s0;
    const float inv_bs = 1.0f / (float)g.bs;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int4* src = part + T.srt_off + s0;
    const int32_t* p = xyz + 3 * T.pt_off;
    auto load = [&](int i) {
        if (!direct) return src[i];
        return make_int4(rel_coord(p[3 * (int64_t)i], T.ox), rel_coord(p[3 * (int64_t)i + 1], T.oy), p[3 * (int64_t)i + 2],
                         (int)(gid ? gid[T.pt_off + i] : (uint32_t)i));
    };
    unsigned bad = 0;        // counted and reported by k_region_count
    auto bin = [&](const int4& v) { return (int)point_bin_est(g, inv_bs, v.x, v.y, bad) & mask; };
    for (int k = tid; k < nb; k += kSortThreads) cnt[k] = 0;
    if (tid < 2) any[tid] = 0;
    __syncthreads();
    const bool held = kHold && n <= kHold * kSortThreads;
    int at[kHold ? kHold : 1];           // bin, and the rank inside it above bit 12
    if (held) {
#pragma unroll
        for (int b = 0; b < kHold; b += kB) {
            int4 v[kB];
#pragma unroll
            for (int k = 0; k < kB; ++k)
                if ((b + k) * kSortThreads + tid < n) v[k] = load((b + k) * kSortThreads + tid);
#pragma unroll
            for (int k = 0; k < kB; ++k)
                if ((b + k) * kSortThreads + tid < n) {
                    const int c = bin(v[k]);
                    at[b + k] = c | (atomicAdd(&cnt[c], 1) << 12);
                }
        }
    } else {
        for (int b = tid; b < n; b += kB * kSortThreads) {
            int4 v[kB];
#pragma unroll
            for (int k = 0; k < kB; ++k)
                if (b + k * kSortThreads < n) v[k] = load(b + k * kSortThreads);
#pragma unroll
            for (int k = 0; k < kB; ++k)
                if (b + k * kSortThreads < n) atomicAdd(&cnt[bin(v[k])], 1);
        }
    }
    __syncthreads();
    // exclusive scan of the nb counts, nb / kSortThreads to a thread
    constexpr int per = nb / kSortThreads;
    int sum = 0;
    for (int k = 0; k < per; ++k) sum += cnt[tid * per + k];
    int x = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) { const int y = __shfl_up_sync(0xffffffffu, x, o); if (lane >= o) x += y; }
    if (lane == 31) wsum[warp] = x;
    __syncthreads();
    int w = lane < kSortThreads / 32 ? wsum[lane] : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) { const int y = __shfl_up_sync(0xffffffffu, w, o); if (lane >= o) w += y; }
    int run = x - sum + (warp ? __shfl_sync(0xffffffffu, w, warp - 1) : 0);
    for (int k = 0; k < per; ++k) {
        const int c = cnt[tid * per + k];
        cnt[tid * per + k] = run;
        run += c;
    }
    if (tid == 0) cnt[nb] = n;
    __syncthreads();
    int* start = start_all + T.bin_off + (int64_t)r * nb;
    uint32_t* bm = (uint32_t*)(bmask + T.blk_off) + ((int64_t)r * nb >> 5);
    for (int k = tid; k < nb; k += kSortThreads) {
        const int c = cnt[k];
        start[k] = s0 + c;
        const unsigned m = __ballot_sync(0xffffffffu, cnt[k + 1] != c);
        if (lane == 0) {
            bm[k >> 5] = m;
            if (m) atomicOr(&any[k >> 11], 1u << ((k >> 6) & 31));
        }
    }
    if (r == nreg - 1 && tid == 0) start[nb] = (int)T.npts;
    __syncthreads();
    if (tid == 0) {
        uint64_t* sm = smask + T.sup_off;
        if (kRsh == 12) sm[r] = (uint64_t)any[0] | ((uint64_t)any[1] << 32);
        else ((unsigned char*)sm)[r] = (unsigned char)any[0];   // a strip is one row of eight blocks
    }
    int4* out = sorted + T.srt_off + s0;
    if (held) {
#pragma unroll
        for (int b = 0; b < kHold; b += kB) {
            int4 v[kB];
#pragma unroll
            for (int k = 0; k < kB; ++k)
                if ((b + k) * kSortThreads + tid < n) v[k] = load((b + k) * kSortThreads + tid);
#pragma unroll
            for (int k = 0; k < kB; ++k)
                if ((b + k) * kSortThreads + tid < n) out[cnt[at[b + k] & 4095] + (at[b + k] >> 12)] = v[k];
        }
    } else {
        for (int b = tid; b < n; b += kB * kSortThreads) {
            int4 v[kB];
#pragma unroll
            for (int k = 0; k < kB; ++k)
                if (b + k * kSortThreads < n) v[k] = load(b + k * kSortThreads);
#pragma unroll
            for (int k = 0; k < kB; ++k)
                if (b + k * kSortThreads < n) out[atomicAdd(&cnt[bin(v[k])], 1)] = v[k];
        }
    }
}

// ---- binning with per-bin global counters: the same result without the
// partition's copy of the points, for callers whose scratch limit leaves no
// room for it ----

// Counting-sort pass 1: per-bin counts, with reductions whose result is not
// returned (no round trip per point).  with_bbox: also the bounding box and
// range checks of k_bbox (batches, whose bin grids are planned before any
// point is seen, skip k_bbox).
__global__ void __launch_bounds__(kChunkThreads) k_bin_count(BatchTables bt, const int32_t* __restrict__ xyz,
                                                   int* __restrict__ cnt, Scalars* sc, BatchCounters* ctr,
                                                   int with_bbox) {
    const int t = find_tile(bt.chunk_base, bt.ntiles, blockIdx.x);
    const TileParams& T = bt.tiles[t];
    const int64_t c0 = (int64_t)(blockIdx.x - __ldg(&bt.chunk_base[t])) * bt.chunk;
    const int64_t c1 = c0 + bt.chunk < T.npts ? c0 + bt.chunk : T.npts;
    const int32_t* p = xyz + 3 * T.pt_off;
    int* c = cnt + T.bin_off;
    unsigned bad = 0;
    BBoxAcc acc;
    for (int64_t i = c0 + threadIdx.x; i < c1; i += blockDim.x) {
        const int xr = p[3 * i], yr = p[3 * i + 1];
        if (with_bbox) bbox_point(xr, yr, p[3 * i + 2], acc);
        const int64_t id = point_bin_checked(T.bg, rel_coord(xr, T.ox), rel_coord(yr, T.oy), bad);
        atomicAdd(&c[id], 1);
    }
    if (with_bbox) bbox_flush(T, acc, sc + t, ctr);
    if (__any_sync(0xffffffffu, bad) && (threadIdx.x & 31) == 0) atomicOr(&ctr->err, kErrRange);
}

// Counting-sort pass 3: each point takes a slot of its bin by counting the
// bin's count down (cnt ends at zero), at start[bin] + the count taken - 1.
// The order of the points inside a bin is therefore arbitrary, which no
// result depends on: every comparison of sites orders them by (distance,
// gid, z), never by position.
__global__ void __launch_bounds__(kChunkThreads) k_bin_scatter(BatchTables bt, const int32_t* __restrict__ xyz,
                                                     const uint32_t* __restrict__ gid, const int* __restrict__ start,
                                                     int* __restrict__ cnt, int4* __restrict__ sorted) {
    const int t = find_tile(bt.chunk_base, bt.ntiles, blockIdx.x);
    const TileParams& T = bt.tiles[t];
    const int64_t c0 = (int64_t)(blockIdx.x - __ldg(&bt.chunk_base[t])) * bt.chunk;
    const int64_t c1 = c0 + bt.chunk < T.npts ? c0 + bt.chunk : T.npts;
    const int32_t* p = xyz + 3 * T.pt_off;
    const int* st = start + T.bin_off;
    int* c = cnt + T.bin_off;
    int4* out = sorted + T.srt_off;
    unsigned bad = 0;
    for (int64_t i = c0 + threadIdx.x; i < c1; i += blockDim.x) {
        const int xr = rel_coord(p[3 * i], T.ox), yr = rel_coord(p[3 * i + 1], T.oy);
        const int64_t id = point_bin_checked(T.bg, xr, yr, bad);
        const int pos = st[id] + atomicSub(&c[id], 1) - 1;
        const uint32_t g = gid ? gid[T.pt_off + i] : (uint32_t)i;
        out[pos] = make_int4(xr, yr, p[3 * i + 2], (int)g);
    }
}

// ---- exclusive scan of each tile's bin counts (three passes, 4096 per block) ----

template <typename V>
__device__ __forceinline__ V block_exclusive_sum(V v, V* wsum, V& total, int tid) {
    // 256 threads (8 warps); tid is the linear thread index in the block
    const int lane = tid & 31, warp = tid >> 5;
    V x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        V y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) wsum[warp] = x;
    __syncthreads();
    if (warp == 0) {
        V w = lane < 8 ? wsum[lane] : V(0);
#pragma unroll
        for (int o = 1; o < 8; o <<= 1) {
            V y = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) w += y;
        }
        if (lane < 8) wsum[lane] = w;
    }
    __syncthreads();
    total = wsum[7];
    const V excl = x - v + (warp ? wsum[warp - 1] : V(0));
    __syncthreads();
    return excl;
}

__global__ void __launch_bounds__(kScanThreads) k_scan_partial(BatchTables bt, const int* __restrict__ cnt,
                                                               int* __restrict__ bsum) {
    __shared__ int wsum[8];
    const int t = find_tile(bt.scan_base, bt.ntiles, blockIdx.x);
    const TileParams& T = bt.tiles[t];
    const int64_t m = T.bg.nbins + 1;
    const int64_t base = (int64_t)(blockIdx.x - __ldg(&bt.scan_base[t])) * kScanTile;
    const int* c = cnt + T.bin_off;
    int s = 0;
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
        const int64_t idx = base + k * kScanThreads + threadIdx.x;
        if (idx < m) s += c[idx];
    }
    int total;
    block_exclusive_sum(s, wsum, total, (int)threadIdx.x);
    if (threadIdx.x == 0) bsum[blockIdx.x] = total;
}

// One block per tile: exclusive scan of the tile's block sums, in place.
__global__ void __launch_bounds__(1024) k_scan_bsum(BatchTables bt, int* __restrict__ bsum) {
    __shared__ int wsum[32];
    const int t = blockIdx.x;
    const int b0g = __ldg(&bt.scan_base[t]), nb = __ldg(&bt.scan_base[t + 1]) - b0g;
    int* bs = bsum + b0g;
    const int per = (nb + 1023) / 1024;
    const int b0 = threadIdx.x * per;
    int s = 0;
    for (int k = 0; k < per; ++k) if (b0 + k < nb) s += bs[b0 + k];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int x = s;
    for (int o = 1; o < 32; o <<= 1) { int y = __shfl_up_sync(0xffffffffu, x, o); if (lane >= o) x += y; }
    if (lane == 31) wsum[warp] = x;
    __syncthreads();
    if (warp == 0) {
        int w = wsum[lane];
        for (int o = 1; o < 32; o <<= 1) { int y = __shfl_up_sync(0xffffffffu, w, o); if (lane >= o) w += y; }
        wsum[lane] = w;
    }
    __syncthreads();
    int run = x - s + (warp ? wsum[warp - 1] : 0);
    for (int k = 0; k < per; ++k)
        if (b0 + k < nb) { const int v = bs[b0 + k]; bs[b0 + k] = run; run += v; }
}

__global__ void __launch_bounds__(kScanThreads) k_scan_final(BatchTables bt, const int* __restrict__ cnt,
                                                             const int* __restrict__ bsum, int* __restrict__ start) {
    __shared__ int tile[kScanTile];
    __shared__ int wsum[8];
    const int t = find_tile(bt.scan_base, bt.ntiles, blockIdx.x);
    const TileParams& T = bt.tiles[t];
    const int64_t m = T.bg.nbins + 1;
    const int64_t base = (int64_t)(blockIdx.x - __ldg(&bt.scan_base[t])) * kScanTile;
    const int* c = cnt + T.bin_off;
    int* st = start + T.bin_off;
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
        const int li = k * kScanThreads + threadIdx.x;
        const int64_t idx = base + li;
        tile[li] = idx < m ? c[idx] : 0;
    }
    __syncthreads();
    int v[kScanItems];
    int s = 0;
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) { v[k] = tile[threadIdx.x * kScanItems + k]; s += v[k]; }
    int total;
    int run = block_exclusive_sum(s, wsum, total, (int)threadIdx.x) + bsum[blockIdx.x];
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) { tile[threadIdx.x * kScanItems + k] = run; run += v[k]; }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
        const int li = k * kScanThreads + threadIdx.x;
        const int64_t idx = base + li;
        if (idx < m) st[idx] = tile[li];
    }
}

// ---------------------------------------------------------------------------
// occupancy masks and the nearest non-empty block map
// ---------------------------------------------------------------------------

// One warp per block (bit l = bin l of the block is non-empty).
__global__ void __launch_bounds__(256) k_block_masks(BatchTables bt, const int* __restrict__ start,
                                                     uint64_t* __restrict__ bmask) {
    const int64_t w = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (w >= __ldg(&bt.blk_base[bt.ntiles])) return;
    const int t = find_tile(bt.blk_base, bt.ntiles, w);
    const TileParams& T = bt.tiles[t];
    const int64_t k = w - T.blk_off;
    const int* s = start + T.bin_off + (k << 6);
    const bool lo = s[lane + 1] != s[lane];
    const bool hi = s[lane + 33] != s[lane + 32];
    const unsigned mlo = __ballot_sync(0xffffffffu, lo), mhi = __ballot_sync(0xffffffffu, hi);
    if (lane == 0) bmask[w] = (uint64_t)mlo | ((uint64_t)mhi << 32);
}

// One warp per superblock (bit m = block m of the superblock is non-empty).
__global__ void __launch_bounds__(256) k_super_masks(BatchTables bt, const uint64_t* __restrict__ bmask,
                                                     uint64_t* __restrict__ smask) {
    const int64_t w = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (w >= __ldg(&bt.sup_base[bt.ntiles])) return;
    const int t = find_tile(bt.sup_base, bt.ntiles, w);
    const TileParams& T = bt.tiles[t];
    const uint64_t* b = bmask + T.blk_off + ((w - T.sup_off) << 6);
    const unsigned mlo = __ballot_sync(0xffffffffu, b[lane] != 0), mhi = __ballot_sync(0xffffffffu, b[lane + 32] != 0);
    if (lane == 0) smask[w] = (uint64_t)mlo | ((uint64_t)mhi << 32);
}

// Nearest non-empty block map, exact in block-centre distance: per block
// row the nearest non-empty column (forward and backward sweep), then per
// block the best row found by walking rows outward until the row offset
// alone exceeds the best distance.  near = bmask index of the chosen block
// within the tile, -1 when the tile has no points.
// One warp per block row, 32 blocks at a time: a ballot of the non-empty ones
// gives each block the nearest on either side (a thread per row, walking its
// blocks one by one, took 90 us for 20 M points on 4096^2 cells).
__global__ void __launch_bounds__(128) k_block_rows(BatchTables bt, const uint64_t* __restrict__ bmask,
                                                    int* __restrict__ rownear) {
    chained();
    const int r = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (r >= __ldg(&bt.row1_base[bt.ntiles])) return;
    const int t = find_tile(bt.row1_base, bt.ntiles, r);
    const TileParams& T = bt.tiles[t];
    const BinGrid g = T.bg;
    const int n1x = g.nbx >> 3;                          // a multiple of 8
    const int cy = r - __ldg(&bt.row1_base[t]);
    const uint64_t* bm = bmask + T.blk_off;
    int* row = rownear + T.blk_off + (int64_t)cy * n1x;
    int last = -1;                                       // nearest non-empty column to the left
    for (int c0 = 0; c0 < n1x; c0 += 32) {
        const int cx = c0 + lane;
        const unsigned m = __ballot_sync(0xffffffffu, cx < n1x && bm[block_index(g, cx, cy)]);
        const unsigned below = m & (0xffffffffu >> (31 - lane));
        if (cx < n1x) row[cx] = below ? c0 + 31 - __clz(below) : last;
        if (m) last = c0 + 31 - __clz(m);
    }
    last = -1;                                           // and to the right
    for (int c0 = (n1x - 1) & ~31; c0 >= 0; c0 -= 32) {
        const int cx = c0 + lane;
        const unsigned m = __ballot_sync(0xffffffffu, cx < n1x && bm[block_index(g, cx, cy)]);
        const unsigned above = m & (0xffffffffu << lane);
        const int right = above ? c0 + __ffs(above) - 1 : last;
        if (cx < n1x) {
            const int l = row[cx];                       // written by this lane
            if (right >= 0 && (l < 0 || right - cx < cx - l)) row[cx] = right;
        }
        if (m) last = c0 + __ffs(m) - 1;
    }
}

// Also starts the raster tiles' largest R2 at none (the binning's grouped
// points lay over them until now).
constexpr int kNearMaskCols = 8;     // superblock columns up to which k_block_near needs no row sweep
__global__ void k_block_near(BatchTables bt, const uint64_t* __restrict__ smask, const int* __restrict__ rownear,
                             int64_t* __restrict__ near, int* __restrict__ rtmax) {
    chained();
    const int64_t w = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    for (int64_t k = w; k < bt.rt_base[bt.ntiles]; k += (int64_t)gridDim.x * blockDim.x) rtmax[k] = -1;
    if (w >= __ldg(&bt.blk_base[bt.ntiles])) return;
    const int t = find_tile(bt.blk_base, bt.ntiles, w);
    const TileParams& T = bt.tiles[t];
    if (T.npts == 0) {   // no row sweep ran for a tile without points
        near[w] = -1;
        return;
    }
    const int n1x = T.bg.nbx >> 3, n1y = T.bg.nby >> 3;
    const int64_t k = w - T.blk_off;
    const int cx = (int)(k % n1x), cy = (int)(k / n1x);
    const int* rn = rownear + T.blk_off;
    if (T.bg.n2x <= kNearMaskCols) {
        // a row of at most 64 blocks is one word, put together from the
        // superblocks' masks: no row sweep
        long long best = LLONG_MAX;
        int bxn = -1, byn = -1;
        for (int d = 0; d < n1y && (long long)d * d <= best; ++d)
            for (int sgn = -1; sgn <= 1; sgn += 2) {
                const int y = cy + sgn * d;
                if ((d == 0 && sgn > 0) || y < 0 || y >= n1y) continue;
                uint64_t row = 0;
                for (int sx = 0; sx < T.bg.n2x; ++sx)
                    row |= ((__ldg(&smask[T.sup_off + (y >> 3) * T.bg.n2x + sx]) >> (8 * (y & 7))) & 0xFF) << (8 * sx);
                const uint64_t below = row & (~0ull >> (63 - cx)), above = row & (~0ull << cx);
                int x = -1;
                if (below) x = 63 - __clzll((long long)below);
                if (above) {
                    const int a = ffs64(above);
                    if (x < 0 || a - cx < cx - x) x = a;
                }
                if (x < 0) continue;
                const long long v = (long long)(x - cx) * (x - cx) + (long long)d * d;
                if (v < best) { best = v; bxn = x; byn = y; }
            }
        near[w] = bxn >= 0 ? block_index(T.bg, bxn, byn) : -1;
        return;
    }
    long long best = LLONG_MAX;
    int bxn = -1, byn = -1;
    for (int d = 0; d < n1y; ++d) {
        if ((long long)d * d > best) break;
        for (int sgn = -1; sgn <= 1; sgn += 2) {
            if (d == 0 && sgn > 0) continue;
            const int y = cy + sgn * d;
            if (y < 0 || y >= n1y) continue;
            const int x = rn[(int64_t)y * n1x + cx];
            if (x < 0) continue;
            const long long v = (long long)(x - cx) * (x - cx) + (long long)d * d;
            if (v < best) { best = v; bxn = x; byn = y; }
        }
    }
    near[w] = bxn >= 0 ? block_index(T.bg, bxn, byn) : -1;
}

// ---------------------------------------------------------------------------
// nearest site per raster pixel
// ---------------------------------------------------------------------------

// Records a settled pixel: its record and (optionally) its site.
__device__ __forceinline__ void settle_pixel(const TileParams& T, int i, int j, const Best& b, int R2,
                                             int2* __restrict__ pix, uint32_t* __restrict__ site) {
    const int64_t o = (int64_t)j * T.rw + i;
    pix[T.pix_off + o] = make_int2(b.z, R2);
    if (site && T.site_off >= 0) site[T.site_off + o] = b.gid;
}

// Statistics of settled pixels, accumulated per thread and flushed once per
// warp: span-path pixels and their spans, the largest R2, and the candidate
// distance evaluations made (counted into evals_dense or evals_far).
struct StatAcc {
    unsigned big = 0, spans = 0, nev = 0;
    int mx = -1;
    __device__ __forceinline__ void add(const TileParams& T, int R2, int n) {
        if (R2 > T.rs * T.rs) {
            big += 1u;
            spans += 2u * (unsigned)isqrt_i32(R2) + 1u;
        }
        mx = R2 > mx ? R2 : mx;
        nev += (unsigned)n;
    }
    __device__ __forceinline__ void flush(Scalars* __restrict__ s, int slot, bool far_pass) {
        const unsigned nbig = __reduce_add_sync(0xffffffffu, big);
        const unsigned nsp = __reduce_add_sync(0xffffffffu, spans);
        const unsigned nv = __reduce_add_sync(0xffffffffu, nev);
        const int m = __reduce_max_sync(0xffffffffu, mx);
        if ((threadIdx.x & 31) == 0) {
            slot &= kStatSlots - 1;
            if (nbig) {
                atomicAdd(&s->big_pixels[slot], (unsigned long long)nbig);
                atomicAdd(&s->spans[slot], (unsigned long long)nsp);
            }
            if (nv) atomicAdd(far_pass ? &s->evals_far[slot] : &s->evals_dense[slot], (unsigned long long)nv);
            if (m >= 0) atomicMax(&s->max_r2[slot], m);
        }
    }
};

// One group of the far worklist: 32 neighbouring pixels of one tile (an 8 x 4
// block or a 32 x 1 row, far_lane), from raster pixel (i0, j0).  idx: per
// lane the sorted-array position of the best site so far (-1 = none,
// kFarIdle = settled or outside the raster).
struct FarGroup {
    int tile, rt, i0, j0;        // rt: raster tile (launch index) the group lies in
    int idx[32];
};
constexpr int kFarIdle = -2;

// Pixel of a group's lane relative to the group's first one.
__device__ __forceinline__ void far_lane(int far_blocks, int lane, int& di, int& dj) {
    di = far_blocks ? lane & 7 : lane;
    dj = far_blocks ? lane >> 3 : 0;
}

// The worklist buffer (kFarSlotBytes per pixel of the padded rasters) holds
// the far groups, then one int per raster tile (the largest R2 of its
// pixels) and the span work items (at most kSpanItemsPerTile per raster tile).
constexpr int kFarSlotBytes = 16;
constexpr int kSpanItemsPerTile = 64;
struct FarLayout {
    FarGroup* groups;
    int* rtmax;
    int2* items;
};
__host__ __device__ inline FarLayout far_layout(void* base, int64_t slots, int64_t nrt) {
    unsigned char* b = (unsigned char*)base;
    FarLayout L;
    L.groups = (FarGroup*)b;
    b += (sizeof(FarGroup) * (slots / 32) + 255) & ~(size_t)255;
    L.rtmax = (int*)b;
    b += (sizeof(int) * nrt + 255) & ~(size_t)255;
    L.items = (int2*)b;
    return L;
}
// groups 4.5 B per slot, rtmax 4 B and items 512 B per 2048 slots, two roundings
static_assert(sizeof(FarGroup) == 144 && 2048 / 32 * sizeof(FarGroup) + 2 * 260 + 8 * kSpanItemsPerTile <=
                  2048 * kFarSlotBytes, "the worklist buffer holds its three parts");

// R2 of a pixel record that the ring search left unsettled (the far pass
// overwrites it); real records hold R2 >= -1.
constexpr int kPixFar = -2;
constexpr int kFarBlocksDefault = 1;   // far groups of 8 x 4 pixels

// Dense pass.  One CTA (256 threads) per 32 x kTileY raster tile of a work
// package, or per 1/split of its rows; each warp takes 8 x 4 blocks of
// pixels.  The block's bin window (bin rings of every pixel) is staged in
// shared memory and the rings are searched there; windows too large for
// shared memory use the global arrays.  Pixels the rings do not settle go to
// the far worklist, 32 to a group: the warp's 8 x 4 block, or a 32 x 1 row.
// With no points every pixel is settled as "no site".
//
// Bound by instruction issue (79 % of the issue slots; 4096^2, 20 M points:
// 1400 warp instructions per 32 pixels, a third of them staging and settling,
// the rest the candidate loops at 22 of 32 lanes).  Visiting a row or column
// of bins only while the gap to it allows a nearer site, two candidates per
// loop turn, quotients from float estimates and bands sized from the plan took
// it from 1074 to 808 us there, and three CTAs per SM with windows of 3584
// points in place of four with 2560 (taller bands, fewer points staged twice)
// to 752 us (1024 mixed tiles 9.97 -> 9.33 ms).  split: a launch with too few
// raster tiles to fill the SMs twice (eight CTAs per SM) cuts them into strips
// of down to 8 rows; the 512^2 case (128 tiles) 66 -> 24 us, the 96 x 80 case (6
// tiles) 41 -> 10 us.
template <bool kDup>
__global__ void __launch_bounds__(256, 3) k_near_dense(BatchTables bt, const int4* __restrict__ pts_all,
                                                       const int* __restrict__ start_all, int2* __restrict__ pix,
                                                       uint32_t* __restrict__ site, FarLayout far,
                                                       Scalars* __restrict__ sc, BatchCounters* __restrict__ ctr,
                                                       int far_blocks, int band0, int split) {
    chained();
    extern __shared__ int4 smem[];
    int4* s_pts = smem;
    int* s_lstart = (int*)(smem + kWinMaxPts + 1);
    int* s_gstart = s_lstart + kWinMaxBins + 1;
    __shared__ int s_rowbase[kWinMaxRows];
    __shared__ int s_max[8];
    const int tid = threadIdx.x;
    const int rt = blockIdx.x / split;
    const int t = find_tile(bt.rt_base, bt.ntiles, rt);
    const TileParams T = bt.tiles[t];   // by value: what the loops use stays in registers
    const BinGrid g = T.bg;
    const float inv_bs = 1.0f / (float)g.bs, inv_cs2 = 1.0f / ((float)T.cs * (float)T.cs);
    const int4* pts = pts_all + T.srt_off;
    const int* start = start_all + T.bin_off;
    const int lt = rt - __ldg(&bt.rt_base[t]);
    const int ntx = (T.rw + kTileX - 1) / kTileX;
    const int rows = kTileY / split;
    const int i0 = (lt % ntx) * kTileX, j0 = (lt / ntx) * kTileY + (blockIdx.x - rt * split) * rows;
    if (j0 >= T.rh) return;
    const int warp = tid >> 5, lane = tid & 31;
    // a warp's 8 x 4 pixels inside each 32 x 8 strip
    const int bi = i0 + (warp & 3) * 8, i = bi + (lane & 7);
    const int sj = (warp >> 2) * 4;
    // the tile's rows go in bands, each with its own staged window: band0
    // rows (8, 16, 32 or 64: the shape of the pixel block that shares one
    // window, a tuning choice) when that window fits shared memory, else
    // halves, down to 8 rows
    StatAcc acc;
    int band = min(min(band0, rows), T.band);
    for (int jb = 0; jb < rows && j0 + jb < T.rh; jb += band) {
    int wx0 = 0, wy0 = 0, wnx = 0, wny = 0;
    bool staged = false;
    while (T.npts > 0) {
        tile_window(T, i0, j0 + jb, band, wx0, wy0, wnx, wny);
        const int nwb = wnx * wny;
        if (nwb > kWinMaxBins || wny > kWinMaxRows) {
            if (band > 8) { band >>= 1; continue; }
            break;
        }
        {
            // each window bin's global start and end, copied asynchronously
            // (all of a band's copies in flight at once; a thread later reads
            // only the entries it copied itself): warp w takes window rows w,
            // w+8, ...; lanes take columns
            for (int r = warp; r < wny; r += 8)
                for (int c = lane; c < wnx; c += 32) {
                    const int64_t id = bin_id(g, wx0 + c, wy0 + r);
                    __pipeline_memcpy_async(&s_gstart[r * wnx + c], &start[id], sizeof(int));
                    __pipeline_memcpy_async(&s_lstart[r * wnx + c], &start[id + 1], sizeof(int));
                }
            __pipeline_commit();
            __pipeline_wait_prior(0);
            // per-bin counts -> local starts, with a warp scan along the row
            for (int r = warp; r < wny; r += 8) {
                int rowsum = 0;
                for (int c0 = 0; c0 < wnx; c0 += 32) {
                    const int c = c0 + lane;
                    int cnt = 0;
                    if (c < wnx) cnt = s_lstart[r * wnx + c] - s_gstart[r * wnx + c];
                    int x = cnt;
#pragma unroll
                    for (int o = 1; o < 32; o <<= 1) {
                        const int y = __shfl_up_sync(0xffffffffu, x, o);
                        if (lane >= o) x += y;
                    }
                    if (c < wnx) s_lstart[r * wnx + c] = rowsum + x - cnt;
                    rowsum += __shfl_sync(0xffffffffu, x, 31);
                }
                if (lane == 0) s_rowbase[r] = rowsum;
            }
            __syncthreads();
            int total = 0;
            for (int r0 = 0; r0 < wny; r0 += 32)
                total += __reduce_add_sync(0xffffffffu, r0 + lane < wny ? s_rowbase[r0 + lane] : 0);
            if (total > kWinMaxPts && band > 8) {     // too many points: a shorter band
                band >>= 1;
                __syncthreads();
                continue;
            }
            staged = total <= kWinMaxPts;
            if (staged) {
                // every warp scans the row sums and places its own rows: adds
                // the row's base to the bins' starts and copies the points
                // (asynchronous 16-byte copies, all in flight before one
                // wait); the bins of one window row inside one block are
                // consecutive in both layouts, lanes striding over the points
                const int cb0 = wx0 >> 3, cb1 = (wx0 + wnx - 1) >> 3;
                int base = 0;
                for (int r0 = 0; r0 < wny; r0 += 32) {
                    const int v = r0 + lane < wny ? s_rowbase[r0 + lane] : 0;
                    int x = v;
#pragma unroll
                    for (int o = 1; o < 32; o <<= 1) {
                        const int y = __shfl_up_sync(0xffffffffu, x, o);
                        if (lane >= o) x += y;
                    }
                    for (int r = r0 + warp; r < min(r0 + 32, wny); r += 8) {
                        const int rb = base + __shfl_sync(0xffffffffu, x - v, r - r0);
                        const int re = base + __shfl_sync(0xffffffffu, x, r - r0);
                        int* ls = s_lstart + r * wnx;
                        for (int c = lane; c < wnx; c += 32) ls[c] += rb;
                        __syncwarp();
                        for (int cb = cb0; cb <= cb1; ++cb) {
                            const int xa = max(cb * 8 - wx0, 0), xb = cb * 8 + 8 - wx0;
                            const int l0 = ls[xa], l1 = xb < wnx ? ls[xb] : re;
                            const int4* src = pts + (s_gstart[r * wnx + xa] - l0);
                            for (int q = l0 + lane; q < l1; q += 32) {
                                __pipeline_memcpy_async(&s_pts[q], &src[q], sizeof(int4));
                                // a copy of the last point follows it (scan_local32)
                                if (q == total - 1) __pipeline_memcpy_async(&s_pts[total], &src[q], sizeof(int4));
                            }
                        }
                    }
                    base += __shfl_sync(0xffffffffu, x, 31);
                }
                if (tid == 0) s_lstart[nwb] = total;
                __pipeline_commit();
                __pipeline_wait_prior(0);
            }
            __syncthreads();
        }
        break;
    }
    const bool fits32 = staged && window_fits32(g, BinWindow{wx0, wy0, wnx, wny, s_lstart, s_gstart, s_pts});
#pragma unroll 1
    for (int sub = 0; sub < band / 8 && j0 + jb + 8 * sub < T.rh; ++sub) {
    const int bj = j0 + jb + 8 * sub + sj, j = bj + (lane >> 3);
    const bool valid = i < T.rw && j < T.rh;
    int R2 = -1;
    bool far_pixel = false;
    Best b{LLONG_MAX, 0xFFFFFFFFu, INT_MAX, -1, 0};
    if (valid) {
        if (T.npts > 0) {
            const int px = (T.rx0 + i) * T.cs, py = (T.ry0 + j) * T.cs;
            bool done;
            if (staged) {
                const BinWindow w{wx0, wy0, wnx, wny, s_lstart, s_gstart, s_pts};
                done = fits32 ? search_window32<kDup>(g, w, inv_bs, px, py, b) : search_window_fast(g, w, px, py, b);
                if (!done) b.idx = window_global_index(w, b.idx);
            } else {
                done = search_bins(g, pts, start, px, py, b);
            }
            if (done) {
                R2 = fits32 && T.cs < (1 << 15) ? r2_of32((unsigned)b.d2, T.cs, inv_cs2, T.r2cap)
                                                : r2_of(b.d2, (long long)T.cs * T.cs, T.r2cap);
                settle_pixel(T, i, j, b, R2, pix, site);
            } else {
                far_pixel = true;
            }
        } else {
            const int64_t o = (int64_t)j * T.rw + i;
            pix[T.pix_off + o] = make_int2(0, -1);
            if (site && T.site_off >= 0) site[T.site_off + o] = 0xFFFFFFFFu;
        }
    }
    if (far_blocks) {
        // a block with any unsettled pixel is one group of the worklist
        if (__any_sync(0xffffffffu, far_pixel)) {
            int base = 0;
            if (lane == 0) {
                base = atomicAdd(&ctr->nfar, 1);
                *reinterpret_cast<int4*>(&far.groups[base]) = make_int4(t, rt, bi, bj);
            }
            base = __shfl_sync(0xffffffffu, base, 0);
            far.groups[base].idx[lane] = far_pixel ? b.idx : kFarIdle;
        }
    } else if (far_pixel) {
        // marked for the row pass below: the record holds the best site found
        // so far (-1: none) and kPixFar
        pix[T.pix_off + (int64_t)j * T.rw + i] = make_int2(b.idx, kPixFar);
    }
    acc.add(T, R2, b.nev);
    }
    __syncthreads();     // the next band restages the window
    }
    acc.flush(sc + t, blockIdx.x + warp, false);
    // the largest R2 of the pixels settled here, for the span work items (the
    // far pass raises it for the others)
    {
        const int m = __reduce_max_sync(0xffffffffu, acc.mx);
        if (lane == 0) s_max[warp] = m;
        __syncthreads();
        if (tid < 32) {
            const int v = __reduce_max_sync(0xffffffffu, s_max[tid & 7]);
            if (tid == 0 && v >= 0) atomicMax(&far.rtmax[rt], v);
        }
    }
    if (!far_blocks) {
        // worklist in pixel rows: a row with any unsettled pixel is one group
        // (the records written above are visible after the barrier)
        for (int r = warp; r < rows; r += 8) {
            const int ii = i0 + lane, jj = j0 + r;
            bool fp = false;
            int idx = -1;
            if (ii < T.rw && jj < T.rh) {
                const int2 rec = pix[T.pix_off + (int64_t)jj * T.rw + ii];
                fp = rec.y == kPixFar;
                idx = rec.x;
            }
            if (__any_sync(0xffffffffu, fp)) {
                int base = 0;
                if (lane == 0) {
                    base = atomicAdd(&ctr->nfar, 1);
                    *reinterpret_cast<int4*>(&far.groups[base]) = make_int4(t, rt, i0, jj);
                }
                base = __shfl_sync(0xffffffffu, base, 0);
                far.groups[base].idx[lane] = fp ? idx : kFarIdle;
            }
        }
    }
}

// ---------------------------------------------------------------------------
// far pass: the exact nearest site of the pixels that the bin rings leave
// ---------------------------------------------------------------------------

// Number types of the search: D holds a site's squared distance, T the squared
// gaps and bounds that the tests compare.  32-bit where every distance it can
// meet fits (far_fits32); otherwise 64-bit distances, and floats in the tests: a
// gap is exact, its square rounded down, a bound rounded up.  Coordinates in the
// tests are unsigned, relative to the bin grid's origin (below 2^32).
template <bool k32> struct FarNum;
template <> struct FarNum<true> {
    using D = unsigned;
    using T = unsigned;
    static __device__ __forceinline__ T none() { return ~0u; }
    static __device__ __forceinline__ T bound(D d2) { return d2; }
    static __device__ __forceinline__ unsigned bits(T v) { return v; }
    static __device__ __forceinline__ T value(unsigned b) { return b; }
    // gap of [a0, a1] and [b0, b1] (within 2^31 of each other), 0 when they meet
    static __device__ __forceinline__ unsigned gap(unsigned a0, unsigned a1, unsigned b0, unsigned b1) {
        return (unsigned)max(max((int)(b0 - a1), (int)(a0 - b1)), 0);
    }
    // (46340^2 exceeds every bound here)
    static __device__ __forceinline__ T square(unsigned dx, unsigned dy) {
        dx = min(dx, 46340u);
        dy = min(dy, 46340u);
        return dx * dx + dy * dy;
    }
    // at least floor(sqrt(v)) + 1: below 2^31 the estimate is within 0.05
    static __device__ __forceinline__ long long reach(T v) { return (long long)sqrt_est((float)v) + 2; }
};
template <> struct FarNum<false> {
    using D = unsigned long long;
    using T = float;
    static __device__ __forceinline__ T none() { return __uint_as_float(0x7F800000u); }
    static __device__ __forceinline__ T bound(D d2) { return __ull2float_ru(d2); }
    static __device__ __forceinline__ unsigned bits(T v) { return __float_as_uint(v); }   // ordered as the values, none negative
    static __device__ __forceinline__ T value(unsigned b) { return __uint_as_float(b); }
    static __device__ __forceinline__ unsigned gap(unsigned a0, unsigned a1, unsigned b0, unsigned b1) {
        return (max(b0, a1) - a1) + (a0 - min(b1, a0));      // one of them is zero
    }
    static __device__ __forceinline__ T square(unsigned dx, unsigned dy) {
        const float x = __uint2float_rd(dx), y = __uint2float_rd(dy);
        return __fmaf_rd(x, x, __fmul_rd(y, y));
    }
    static __device__ __forceinline__ long long reach(T v) { return reach_of((long long)v) + 1; }
};

// One lane's pixel and best site so far.
template <bool k32>
struct FarLane {
    using D = typename FarNum<k32>::D;
    int px, py;
    D d2;
    uint32_t gid;
    int z, idx;
    __device__ __forceinline__ void consider(const int4 p, int q) {
        D d;
        if (k32) {
            const int dx = p.x - px, dy = p.y - py;
            d = (unsigned)(dx * dx) + (unsigned)(dy * dy);
        } else {
            const int dx = p.x - px, dy = p.y - py;          // |p.x|, |px| < 2^30
            d = (unsigned long long)((long long)dx * dx) + (unsigned long long)((long long)dy * dy);
        }
        if (__builtin_expect(d <= d2, 0)) {
            const uint32_t g = (uint32_t)p.w;
            if (d < d2 || g < gid || (g == gid && p.z < z)) {
                d2 = d;
                gid = g;
                z = p.z;
                idx = q;
            }
        }
    }
};

// A warp leaves a group to the heavy pass once it has searched this many
// blocks for it and more remain: fewer while the groups leave warps without
// work (below four to a warp), and none at all below one group per CTA of the
// heavy pass, which then takes every group.  Beyond 32-bit distances, where a
// CTA's warps share a group less well, a warp goes on as long as kFarKeep groups
// per warp wait to be handed out (2048^2 cells, 0.5 and 8 points per cell around a
// lake 1843 cells wide: far passes 9.6 -> 8.6 and 122 -> 84 ms; going on always
// left long groups to the end, and two smaller lakes took 3.8 in place of 2.2 ms).
constexpr int kFarDefer = 32, kFarDeferFew = 8, kFarKeep = 2;
constexpr int kFarCtasPerSm = 4;
__device__ __forceinline__ bool far_all_heavy(int groups) { return groups <= (int)gridDim.x; }
constexpr int kFarPixels = 32;   // a group spans at most this many cells in x and y

// A warp's buffer of candidate points, and the circles that hold the discs of
// each eighth of its pixels (2 x 2, or 4 x 1 in row groups): centre relative to
// the group's corner and squared radius, rounded up; a negative radius where no
// pixel is active.
struct FarBuf {
    int4 p[32];
    int q[32];
    float4 circle[8];
};

// 32-bit arithmetic serves a search whose bound is `reach` (per lane, the
// largest): a point it evaluates lies in a block some lane's disc touches, so
// within reach + 8 bins + the group's extent of every lane, and that must stay
// within 46340 for the squared distance to fit 32 bits.
__device__ __forceinline__ bool far_fits32(long long reach, int bs, int cs) {
    return reach + 8LL * bs + (long long)kFarPixels * cs <= 46340;
}

// Warp-cooperative exact search for the 32 pixels of one worklist group; every
// lane holds a real site on entry (idle lanes repeat another lane's pixel).
// The group's own superblock comes first, then those within the largest bound,
// one tested per lane; a superblock's blocks, two to a lane, are tested against the
// group's box at once and searched nearest first, so that the bounds tighten
// early; in a block, the bins within the largest bound form one run per row
// (tested the same way), and the runs that some lane's disc touches are ranges
// of points: one point per lane is fetched, and those inside the circle of some
// eighth of the pixels are evaluated by every lane.  Every test is a lower bound
// of the distance against an upper bound of what is sought, so nothing that
// could hold an equally near site is left out.  Uniform control flow in the
// warp.
//
// kCta: the eight warps of a CTA search one group; warp w takes the blocks of
// one residue class, and the lanes' bounds meet in s_bound.  Otherwise the
// search ends with false after `most` blocks if more remain (with `next`, the
// number of groups handed out: only once that has reached `keep`).
template <bool k32, bool kCta>
__device__ __forceinline__ bool far_search(const BinGrid& g, const int4* __restrict__ pts, const int* __restrict__ start,
                                           const uint64_t* __restrict__ bmask, const uint64_t* __restrict__ smask,
                                           FarLane<k32>& b, bool act, unsigned& nev, FarBuf* buf, int far_blocks,
                                           volatile unsigned* s_bound, int most, const int* next, int keep) {
    using N = FarNum<k32>;
    using T = typename N::T;
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned bs = g.bs, u1 = bs * kBinsPerBlockEdge, u2 = bs * kBinsPerSuperEdge;
    const int ox = __reduce_min_sync(full, b.px), oy = __reduce_min_sync(full, b.py);      // the group's corner
    const unsigned X0 = ox - g.gx0, X1 = __reduce_max_sync(full, b.px) - g.gx0;
    const unsigned Y0 = oy - g.gy0, Y1 = __reduce_max_sync(full, b.py) - g.gy0;
    const unsigned px = b.px - g.gx0, py = b.py - g.gy0;
    auto warp_min = [&](T v) { return N::value(__reduce_min_sync(full, N::bits(v))); };
    // lane's bound: nothing farther can matter to it
    auto bound = [&]() -> T {
        const unsigned v = N::bits(N::bound(b.d2));
        return N::value(kCta ? min(v, s_bound[lane]) : v);
    };
    // the circles of the pixels' eighths (far_half, far_circle_r2)
    const int step2 = far_blocks ? 8 : 2;
    float cx0 = act ? (float)(b.px - ox) : 3e38f, cx1 = act ? (float)(b.px - ox) : -3e38f;
    float cy0 = act ? (float)(b.py - oy) : 3e38f, cy1 = act ? (float)(b.py - oy) : -3e38f;
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        const int x = k ? step2 : 1;
        cx0 = fminf(cx0, __shfl_xor_sync(full, cx0, x));
        cx1 = fmaxf(cx1, __shfl_xor_sync(full, cx1, x));
        cy0 = fminf(cy0, __shfl_xor_sync(full, cy0, x));
        cy1 = fmaxf(cy1, __shfl_xor_sync(full, cy1, x));
    }
    const bool none_active = cx0 > cx1;
    const float ccx = 0.5f * (cx0 + cx1), ccy = 0.5f * (cy0 + cy1);
    const float half = far_half(cx1 - cx0, cy1 - cy0, fmaxf((float)(X1 - X0), (float)(Y1 - Y0)));
    const bool writes = !(lane & (1 | step2));
    const int eighth = far_blocks ? ((lane >> 1) & 3) + 4 * (lane >> 4) : lane >> 2;
    T maxd;
    auto new_bounds = [&]() {
        unsigned m = act ? N::bits(bound()) : 0u;
        maxd = N::value(__reduce_max_sync(full, m));
        m = max(m, __shfl_xor_sync(full, m, 1));
        m = max(m, __shfl_xor_sync(full, m, step2));
        const float r2 = far_circle_r2(sqrt_est((float)N::value(m)), half);
        if (writes) buf->circle[eighth] = make_float4(ccx, ccy, none_active ? -1.0f : r2, 0.0f);
        __syncwarp();
    };
    new_bounds();
    // one candidate point to a lane, fetched all at once; those inside a circle
    // are evaluated by every lane
    auto round = [&](int q, bool in) {
        int4 p = make_int4(0, 0, 0, 0);
        if (in) p = __ldg(&pts[q]);
        const float x = (float)(p.x - ox), y = (float)(p.y - oy);
        bool hit = false;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const float4 c = buf->circle[k];
            hit |= far_in_circle(x, y, c.x, c.y, c.z);
        }
        in = in && hit;
        const unsigned got = __ballot_sync(full, in);
        if (!got) return;
        if (in) {
            const int k = __popc(got & ((1u << lane) - 1u));
            buf->p[k] = p;
            buf->q[k] = q;
        }
        __syncwarp();
        const int n = __popc(got);
#pragma unroll 4
        for (int k = 0; k < n; ++k) b.consider(buf->p[k], buf->q[k]);
        nev += n;
        if (kCta) {
            const unsigned v = N::bits(N::bound(b.d2));
            if (v < s_bound[lane]) atomicMin((unsigned*)&s_bound[lane], v);
        }
        new_bounds();                    // (its barrier also ends the buffer's use)
    };
    const long long reach = N::reach(maxd);
    auto cell = [&](long long c, int n) {   // superblock column (row) of a place, clamped to the grid
        return c <= 0 ? 0 : (c >= (long long)n * u2 ? n - 1 : udiv32(c, u2));
    };
    const int sx0 = cell(X0 - reach, g.n2x), sx1 = cell(X1 + reach, g.n2x);
    const int sy0 = cell(Y0 - reach, g.n2y), sy1 = cell(Y1 + reach, g.n2y);
    const int cx = cell(X0, g.n2x), cy = cell(Y0, g.n2y);
    const int nsx = sx1 - sx0 + 1, ns = nsx * (sy1 - sy0 + 1);
    // whether superblock k of the box (row by row; the group's own one: k < 0)
    // can hold points within the bounds
    auto super_at = [&](int k, int& sx, int& sy) {
        sy = k < 0 ? cy : sy0 + (int)((unsigned)k / (unsigned)nsx);
        sx = k < 0 ? cx : sx0 + (int)((unsigned)k % (unsigned)nsx);
        const unsigned SX0 = sx * u2, SY0 = sy * u2;
        return N::square(N::gap(X0, X1, SX0, SX0 + u2 - 1), N::gap(Y0, Y1, SY0, SY0 + u2 - 1)) <= maxd;
    };
    int searched = 0;
    // the group's own superblock first, then the others, one to a lane, and those
    // that remain one by one
    for (int s0 = -1; s0 < ns; s0 += s0 < 0 ? 1 : 32) {
        const int mine = s0 < 0 ? -1 : s0 + lane;
        int mx, my;
        const bool within = mine < ns && (s0 >= 0 || lane == 0) && super_at(mine, mx, my);
        unsigned live = __ballot_sync(full, within && (mine < 0 || mx != cx || my != cy) && __ldg(&smask[my * g.n2x + mx]));
        while (live) {
        int sx, sy;
        const bool still = super_at(s0 < 0 ? -1 : s0 + __ffs(live) - 1, sx, sy);
        live &= live - 1;
        if (!still) continue;            // the bounds have shrunk
        const int sidx = sy * g.n2x + sx;
        const uint64_t sm = __ldg(&smask[sidx]);
        const unsigned SX0 = sx * u2, SY0 = sy * u2;
        // this lane's two blocks: column lane & 7, rows lane >> 3 and + 4
        T key0, key1;
        {
            const unsigned bx = SX0 + (lane & 7) * u1, by = SY0 + (lane >> 3) * u1;
            const unsigned dx = N::gap(X0, X1, bx, bx + u1 - 1);
            key0 = (sm >> lane) & 1 ? N::square(dx, N::gap(Y0, Y1, by, by + u1 - 1)) : N::none();
            key1 = (sm >> (lane + 32)) & 1 ? N::square(dx, N::gap(Y0, Y1, by + 4 * u1, by + 5 * u1 - 1)) : N::none();
            if (kCta) {
                // residue classes of the blocks: neighbouring blocks go to different warps
                const int c = (lane & 7) + 3 * (lane >> 3) + sx + sy;
                if ((c & 7) != warp) key0 = N::none();
                if (((c + 12) & 7) != warp) key1 = N::none();
            }
        }
        // their occupancy and point ranges, all in flight at once
        uint64_t mask0 = 0, mask1 = 0;
        int first0 = 0, last0 = 0, first1 = 0, last1 = 0;
        {
            const int64_t k0 = ((int64_t)sidx << 6) + lane;
            if (key0 <= maxd) {
                mask0 = __ldg(&bmask[k0]);
                first0 = __ldg(&start[k0 << 6]);
                last0 = __ldg(&start[(k0 + 1) << 6]);
            }
            if (key1 <= maxd) {
                mask1 = __ldg(&bmask[k0 + 32]);
                first1 = __ldg(&start[(k0 + 32) << 6]);
                last1 = __ldg(&start[(k0 + 33) << 6]);
            }
        }
        for (;;) {
            const T key = key0 < key1 ? key0 : key1, least = warp_min(key);
            if (least > maxd || least == N::none()) break;
            const int who = __ffs(__ballot_sync(full, key == least)) - 1;
            const int second = __shfl_sync(full, (int)(key0 != least), who);
            if (lane == who) {
                if (second) key1 = N::none(); else key0 = N::none();
            }
            const int m = who + 32 * second;
            const unsigned BX0 = SX0 + (m & 7) * u1, BY0 = SY0 + (m >> 3) * u1;
            // a disc must touch it
            const T bd = bound();
            if (!__any_sync(full, N::square(N::gap(px, px, BX0, BX0 + u1 - 1), N::gap(py, py, BY0, BY0 + u1 - 1)) <= bd)) continue;
            if (!kCta && ++searched > most) {
                if (!next || *(const volatile int*)next >= keep) return false;
                searched = 0;
            }
            const int* st = start + (((int64_t)sidx << 6) + m << 6);
            const int bp0 = __shfl_sync(full, second ? first1 : first0, who);
            const int bp1 = __shfl_sync(full, second ? last1 : last0, who);
            // the block's runs of points, dealt to the lanes one after the other:
            // the whole block when it has few points (its bins are
            // consecutive), else the rows' runs, first to last bin, that some
            // disc touches
            uint64_t run = 0;
            int t0 = 0, t1 = 0, q0 = bp0, q1 = bp1;
            if (bp1 - bp0 > 32) {
                q1 = bp0;
                t0 = __ldg(&st[lane]);
                t1 = __ldg(&st[lane + 32]);
                const unsigned bm0 = __shfl_sync(full, second ? (unsigned)mask1 : (unsigned)mask0, who);
                const unsigned bm1 = __shfl_sync(full, second ? (unsigned)(mask1 >> 32) : (unsigned)(mask0 >> 32), who);
                const unsigned qx = BX0 + (lane & 7) * bs, qy = BY0 + (lane >> 3) * bs;
                const unsigned dx = N::gap(X0, X1, qx, qx + bs - 1);
                const unsigned lo = __ballot_sync(full, N::square(dx, N::gap(Y0, Y1, qy, qy + bs - 1)) <= maxd);
                const unsigned hi = __ballot_sync(full, N::square(dx, N::gap(Y0, Y1, qy + 4 * bs, qy + 5 * bs - 1)) <= maxd);
                run = (uint64_t)(bm0 & lo) | ((uint64_t)(bm1 & hi) << 32);
            }
            for (;;) {
                int fill = 0, q = 0;
                while (fill < 32) {
                    if (q0 == q1) {
                        if (!run) break;
                        const int r = ffs64(run) >> 3;
                        const unsigned bits = (unsigned)(run >> (8 * r)) & 0xFFu;
                        run &= ~(0xFFull << (8 * r));
                        const int a = __ffs(bits) - 1, e = 31 - __clz(bits);
                        const unsigned qx = BX0 + a * bs, qy = BY0 + r * bs;
                        if (!__any_sync(full, N::square(N::gap(px, px, qx, qx + (e - a + 1) * bs - 1),
                                                        N::gap(py, py, qy, qy + bs - 1)) <= bd)) continue;
                        const int ia = 8 * r + a, ie = 8 * r + e + 1;
                        q0 = __shfl_sync(full, ia < 32 ? t0 : t1, ia & 31);
                        q1 = __shfl_sync(full, ie < 32 ? t0 : t1, ie & 31);
                        if (ie == 64) q1 = bp1;
                    }
                    const int take = min(32 - fill, q1 - q0);
                    if ((unsigned)(lane - fill) < (unsigned)take) q = q0 + lane - fill;
                    fill += take;
                    q0 += take;
                }
                if (fill) round(q, lane < fill);
                if (fill < 32) break;
            }
        }
        }
    }
    return true;
}

// A group of the far worklist in one warp's registers: its pixels (idle
// lanes repeat the first active lane's) and the best sites so far.
struct FarWork {
    int t, rt, i, j;
    bool act;
    Best b;
    int px, py;
    unsigned nev;
};

// Loads group k and seeds every lane with a real site: its own best so far,
// the best of the lane that is nearest to one, and points of the non-empty
// bin closest to the group in the non-empty block nearest to it.
__device__ __forceinline__ void far_load(FarWork& w, const BatchTables& bt, const FarLayout& far, int k, int far_blocks,
                                         const int4* __restrict__ pts_all, const int* __restrict__ start_all,
                                         const uint64_t* __restrict__ bmask_all, const int64_t* __restrict__ near_all) {
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int4 head = *reinterpret_cast<const int4*>(&far.groups[k]);
    const int own = far.groups[k].idx[lane];
    w.t = head.x;
    w.rt = head.y;
    const TileParams& T = bt.tiles[w.t];
    const BinGrid g = T.bg;
    const int4* pts = pts_all + T.srt_off;
    const int* start = start_all + T.bin_off;
    w.act = own != kFarIdle;
    int di, dj;
    far_lane(far_blocks, lane, di, dj);
    w.i = head.z + di;
    w.j = head.w + dj;
    const int first = __ffs(__ballot_sync(full, w.act)) - 1;
    w.px = (T.rx0 + w.i) * T.cs;
    w.py = (T.ry0 + w.j) * T.cs;
    const int fx = __shfl_sync(full, w.px, first), fy = __shfl_sync(full, w.py, first);
    if (!w.act) {
        w.px = fx;
        w.py = fy;
    }
    w.b = Best{LLONG_MAX, 0xFFFFFFFFu, INT_MAX, -1, 0};
    w.nev = 0;
    if (own >= 0) {
        consider(w.b, __ldg(&pts[own]), own, w.px, w.py);
        w.nev += 1;
    }
    if (__any_sync(full, own >= 0)) {
        // float order is enough to choose a seed
        const unsigned f = own >= 0 ? __float_as_uint((float)w.b.d2) : 0xffffffffu;
        const int src = __ffs(__ballot_sync(full, f == __reduce_min_sync(full, f))) - 1;
        const int q = __shfl_sync(full, own, src);
        consider(w.b, __ldg(&pts[q]), q, w.px, w.py);
        w.nev += 1;
    }
    const int gx = min(udiv32((long long)fx - g.gx0, g.bs), g.nbx - 1), gy = min(udiv32((long long)fy - g.gy0, g.bs), g.nby - 1);
    const int64_t nb = __ldg(&near_all[T.blk_off + (int64_t)(gy >> 3) * (g.nbx >> 3) + (gx >> 3)]);
    if (nb >= 0) {
        const int sidx = (int)(nb >> 6), m = (int)(nb & 63);
        const uint64_t bm = __ldg(&bmask_all[T.blk_off + nb]);
        // bins relative to the first pixel, in bins: the nearest non-empty one
        const int ox = (sidx % g.n2x) * 64 + (m & 7) * 8 + (lane & 7) - gx;
        const int oy = (sidx / g.n2x) * 64 + (m >> 3) * 8 + (lane >> 3) - gy;
        const float a = (float)ox * (float)ox, c = (float)oy * (float)oy, e = (float)(oy + 4) * (float)(oy + 4);
        const unsigned k0 = (bm >> lane) & 1 ? __float_as_uint(a + c) : 0xffffffffu;
        const unsigned k1 = (bm >> (lane + 32)) & 1 ? __float_as_uint(a + e) : 0xffffffffu;
        const unsigned least = __reduce_min_sync(full, min(k0, k1));
        const int who = __ffs(__ballot_sync(full, min(k0, k1) == least)) - 1;
        const int second = __shfl_sync(full, (int)(k0 != least), who);
        const int64_t id = (nb << 6) + who + 32 * second;
        const int s0 = __ldg(&start[id]), e0 = min(__ldg(&start[id + 1]), s0 + 4);
        w.nev += e0 - s0;
        for (int q = s0; q < e0; ++q) consider(w.b, __ldg(&pts[q]), q, w.px, w.py);
    }
}

template <bool k32, bool kCta>
__device__ __forceinline__ bool far_run(FarWork& w, const TileParams& T, const int4* pts_all, const int* start_all,
                                        const uint64_t* bmask_all, const uint64_t* smask_all, FarBuf* buf, int far_blocks,
                                        volatile unsigned* s_bound, int most, const int* next = nullptr, int keep = 0) {
    FarLane<k32> b{w.px, w.py, (typename FarNum<k32>::D)w.b.d2, w.b.gid, w.b.z, w.b.idx};
    const bool done = far_search<k32, kCta>(T.bg, pts_all + T.srt_off, start_all + T.bin_off, bmask_all + T.blk_off,
                                            smask_all + T.sup_off, b, w.act, w.nev, buf, far_blocks, s_bound, most, next, keep);
    w.b.d2 = (long long)b.d2;
    w.b.gid = b.gid;
    w.b.z = b.z;
    w.b.idx = b.idx;
    return done;
}

__device__ __forceinline__ bool far_small(const FarWork& w, const TileParams& T) {
    const long long r = w.b.d2 < (1LL << 31) ? (long long)sqrt_est((float)w.b.d2) + 2 : LLONG_MAX / 4;
    return __all_sync(0xffffffffu, far_fits32(r, T.bg.bs, T.cs));
}

// The searches beyond 32-bit distances, as functions of their own: inlined, their
// registers cost the 32-bit ones spills.
template <bool kCta>
__device__ __noinline__ bool far_run_wide(FarWork* w, const TileParams* T, const int4* pts_all, const int* start_all,
                                          const uint64_t* bmask_all, const uint64_t* smask_all, FarBuf* buf, int far_blocks,
                                          volatile unsigned* s_bound, int most, const int* next, int keep) {
    return far_run<false, kCta>(*w, *T, pts_all, start_all, bmask_all, smask_all, buf, far_blocks, s_bound, most, next, keep);
}

__device__ __forceinline__ void far_settle(const FarWork& w, const TileParams& T, int2* __restrict__ pix,
                                           uint32_t* __restrict__ site, Scalars* __restrict__ sc, const FarLayout& far,
                                           int slot) {
    int R2 = -1;
    if (w.act) {
        R2 = r2_of(w.b.d2, (long long)T.cs * T.cs, T.r2cap);
        settle_pixel(T, w.i, w.j, w.b, R2, pix, site);
    }
    StatAcc acc;
    acc.add(T, R2, w.act ? (int)w.nev : 0);
    acc.flush(sc + w.t, slot, true);
    const int m = __reduce_max_sync(0xffffffffu, R2);
    if ((threadIdx.x & 31) == 0 && m > T.rs * T.rs) atomicMax(&far.rtmax[w.rt], m);
}

// Far pass over the worklist: one warp per group, handed out by a counter
// (groups differ in cost by orders of magnitude: a lake's centre against its
// shore).  Groups that need more than `most` blocks go, with the sites found so
// far, to the heavy list (in the span items' place, which are listed later; at
// most 64 groups per raster tile).  Groups beyond 32-bit distances (nearest sites
// more than 463 m away at 1 cm) run the wide search, a function of its own: with
// both inlined a warp waited four issue slots for instructions and the 32-bit one
// spilled.  (All such groups on whole CTAs, with 64-bit tests: a 4096^2 tile at
// 0.1 points per cell in millimetres, with lakes, 30.3 ms, now 19.8; 200 mixed
// tiles in millimetres 11.4 ms, now 7.6.)
__global__ void __launch_bounds__(256, 4) k_near_far(BatchTables bt, const int4* __restrict__ pts_all,
                                                     const int* __restrict__ start_all,
                                                     const uint64_t* __restrict__ bmask_all,
                                                     const uint64_t* __restrict__ smask_all,
                                                     const int64_t* __restrict__ near_all,
                                                     FarLayout far, int2* __restrict__ pix,
                                                     uint32_t* __restrict__ site, Scalars* __restrict__ sc,
                                                     BatchCounters* __restrict__ ctr, int far_blocks) {
    chained();
    __shared__ FarBuf s_buf[8];
    const int count = ctr->nfar;
    if (far_all_heavy(count)) return;
    const int lane = threadIdx.x & 31;
    FarBuf* buf = &s_buf[threadIdx.x >> 5];
    const int most = count < (int)gridDim.x * 32 ? kFarDeferFew : kFarDefer;
    int* heavy = (int*)far.items;
    for (;;) {
        int k = 0;
        if (lane == 0) k = atomicAdd(&ctr->far_next, 1);
        k = __shfl_sync(0xffffffffu, k, 0);
        if (k >= count) break;
        FarWork w;
        far_load(w, bt, far, k, far_blocks, pts_all, start_all, bmask_all, near_all);
        const TileParams& T = bt.tiles[w.t];
        bool done;
        if (far_small(w, T)) {
            done = far_run<true, false>(w, T, pts_all, start_all, bmask_all, smask_all, buf, far_blocks, nullptr, most);
        } else {
            FarWork v = w;
            done = far_run_wide<false>(&v, &T, pts_all, start_all, bmask_all, smask_all, buf, far_blocks, nullptr, most, &ctr->far_next, count - kFarKeep * 8 * (int)gridDim.x);
            w = v;
        }
        if (done) {
            far_settle(w, T, pix, site, sc, far, blockIdx.x * 3 + (threadIdx.x >> 5));
        } else {
            if (w.act) far.groups[k].idx[lane] = w.b.idx;
            if (lane == 0) heavy[atomicAdd(&ctr->nheavy, 1)] = k;
        }
    }
}

constexpr int kSpanWindowWords = 4096;      // default: 32 KB per CTA (two int32 arrays)
constexpr int kSpanWindowMaxWords = 26624;  // 208 KB, the most one CTA may take
constexpr int kSpanChunksPerItem = 2;       // window chunks of one span work item, at least

// The grid cells that the discs of one 32 x kTileY raster tile may touch, from
// its largest R2: columns [c0, c1] and rows [r0, r1] of the grid (empty when
// c0 > c1 or r0 > r1), taken `rows` rows at a time by `win_words` cells of
// shared memory (direct: one item, no window), `per` rows to a work item.
struct SpanWindow {
    int c0, c1, r0, r1, W, rows, per;
    int stride;                  // window row stride: W padded to 1 modulo 4 (lanes on successive rows
                                 // whose spans end in one column then fall on different banks)
    bool inside;                 // no span meets the grid's left or right edge
};

__device__ __forceinline__ SpanWindow span_window(const TileParams& T, int lt, int r2, int win_words, bool direct) {
    SpanWindow w;
    const int ntx = (T.rw + kTileX - 1) / kTileX;
    const int i0 = (lt % ntx) * kTileX, j0 = (lt / ntx) * kTileY;
    const int r = isqrt_i32(r2);
    const int xlo = T.rx0 + i0 - r, xhi = T.rx0 + min(i0 + kTileX, T.rw) + r;
    const int ylo = T.ry0 + j0 - r, yhi = T.ry0 + min(j0 + kTileY, T.rh) - 1 + r;
    w.inside = xlo >= 0 && xhi < T.ncols;
    w.c0 = max(xlo, 0);
    w.c1 = min(xhi, T.ncols - 1);
    w.r0 = max(ylo, 0);
    w.r1 = min(yhi, T.nrows - 1);
    w.W = w.c1 - w.c0 + 1;
    w.stride = ((w.W + 2) & ~3) + 1;
    const int n = w.r1 - w.r0 + 1;
    w.rows = w.W > 0 ? (win_words & ~3) / w.stride : 0;
    if (direct || w.rows < 1) {
        w.rows = 0;
        w.per = max(n, 1);
    } else {
        w.rows = min(w.rows, n);
        const int chunks = max((n + w.rows - 1) / w.rows, 1);
        w.per = w.rows * max((chunks + kSpanItemsPerTile - 1) / kSpanItemsPerTile, kSpanChunksPerItem);
    }
    return w;
}

// The window sums z relative to zbase and the counts in two int32 arrays
// (native shared-memory atomics); a window cell receives at most one marker
// per pixel of the tile, so |sum| <= kTileX * kTileY * zabs must stay below
// 2^31.  Otherwise, and without the packed word, every marker goes straight
// to the grid.
__device__ __forceinline__ bool span_direct(const Scalars& s, int zmin, int zmax) {
    const long long zabs = max((long long)zmax - s.zbase, s.zbase - (long long)zmin);
    return !s.packed || zabs >= (1LL << 31) / (kTileX * kTileY);
}

// Lists the span work items of a tile's raster tiles (and layers of them):
// one item per group of window chunks, so that the discs of one raster tile,
// which differ in work by orders of magnitude (a lake's centre against its
// shore), spread over the SMs.
__device__ __forceinline__ void list_span_items(const BatchTables& bt, int t, int layers, bool direct, int win_words,
                                                const FarLayout& far, BatchCounters* ctr) {
    const TileParams& T = bt.tiles[t];
    const int b0 = bt.rt_base[t], nrt = bt.rt_base[t + 1] - b0, rs2 = T.rs * T.rs;
    const int lane = threadIdx.x & 31;
    for (int k0 = 0; k0 < nrt * layers; k0 += blockDim.x) {
        const int k = k0 + threadIdx.x;
        int n = 0;
        SpanWindow w;
        if (k < nrt * layers) {
            const int r2 = __ldcg(&far.rtmax[b0 + k]);
            if (r2 > rs2) {
                w = span_window(T, k % nrt, r2, win_words, direct);
                if (w.c0 <= w.c1 && w.r0 <= w.r1) n = (w.r1 - w.r0 + w.per) / w.per;
            }
        }
        int x = n;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        int base = 0;
        if (lane == 31 && x) base = atomicAdd(&ctr->nspan, x);
        base = __shfl_sync(0xffffffffu, base, 31) + x - n;
        for (int e = 0; e < n; ++e) far.items[base + e] = make_int2(b0 + k, w.r0 + e * w.per);
    }
}

// Per tile: the accumulator form of the span path (see decide_packing) and
// its work items (one block).
__device__ __forceinline__ void decide_tile(const BatchTables& bt, int t, Scalars* sc, const FarLayout& far,
                                            BatchCounters* ctr, int win_words) {
    __shared__ int direct;
    const int l = threadIdx.x;
    const TileParams& T = bt.tiles[t];
    Scalars* s = sc + t;
    if (l < 32) {
        int mx = __ldcg(&s->max_r2[l]);
        mx = __reduce_max_sync(0xffffffffu, mx);
        if (l == 0) {
            int packed, K;
            long long zbase;
            decide_packing(mx, (long long)T.rw * T.rh, s->bbox[4], s->bbox[5], packed, K, zbase);
            s->packed = packed;
            s->kbits = K;
            s->zbase = zbase;
            direct = span_direct(*s, s->bbox[4], s->bbox[5]);
        }
    }
    __syncthreads();
    list_span_items(bt, t, 1, direct != 0, win_words, far, ctr);
}

__global__ void __launch_bounds__(1024) k_decide(BatchTables bt, Scalars* sc, FarLayout far, BatchCounters* ctr,
                                                int win_words) {
    chained();
    decide_tile(bt, blockIdx.x, sc, far, ctr, win_words);
}

// The heavy groups, one CTA of eight warps each.  On the way it clears the span
// words (D, n64 of them) and counts (Dc, n32), which no later phase needs before,
// and with win_words the last block to finish decides the first tile's
// accumulator form and lists its work items (k_decide, for a single work
// package whose raster tiles one block lists quickly).
__global__ void __launch_bounds__(256, 4) k_near_far_heavy(BatchTables bt, const int4* __restrict__ pts_all,
                                                           const int* __restrict__ start_all,
                                                           const uint64_t* __restrict__ bmask_all,
                                                           const uint64_t* __restrict__ smask_all,
                                                           const int64_t* __restrict__ near_all, FarLayout far,
                                                           int2* __restrict__ pix, uint32_t* __restrict__ site,
                                                           Scalars* __restrict__ sc, BatchCounters* __restrict__ ctr,
                                                           int far_blocks, unsigned long long* __restrict__ D, int64_t n64,
                                                           int* __restrict__ Dc, int64_t n32, int win_words) {
    chained();
    for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < n64; k += (int64_t)gridDim.x * blockDim.x) D[k] = 0;
    for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < n32; k += (int64_t)gridDim.x * blockDim.x) Dc[k] = 0;
    __shared__ unsigned s_bound[32];         // each lane's bound, as FarNum::bits gives it
    __shared__ Best s_best[8][32];
    __shared__ FarBuf s_buf[8];
    __shared__ int s_k;
    const bool all = far_all_heavy(ctr->nfar);
    const int count = all ? ctr->nfar : ctr->nheavy;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int* heavy = (const int*)far.items;
    for (;;) {
        __syncthreads();                 // the previous group's readers are done
        if (threadIdx.x == 0) s_k = atomicAdd(&ctr->heavy_next, 1);
        __syncthreads();
        if (s_k >= count) break;
        FarWork w;
        far_load(w, bt, far, all ? s_k : heavy[s_k], far_blocks, pts_all, start_all, bmask_all, near_all);
        const TileParams& T = bt.tiles[w.t];
        const bool small = far_small(w, T);
        if (warp == 0) s_bound[lane] = ~0u;
        __syncthreads();
        if (small) far_run<true, true>(w, T, pts_all, start_all, bmask_all, smask_all, &s_buf[warp], far_blocks, s_bound, 0);
        else far_run<false, true>(w, T, pts_all, start_all, bmask_all, smask_all, &s_buf[warp], far_blocks, s_bound, 0);
        w.b.nev = (int)w.nev;
        s_best[warp][lane] = w.b;
        __syncthreads();
        if (warp == 0) {
            for (int v = 1; v < 8; ++v) {
                const Best o = s_best[v][lane];
                w.nev += (unsigned)o.nev;
                if (o.d2 < w.b.d2 || (o.d2 == w.b.d2 && (o.gid < w.b.gid || (o.gid == w.b.gid && o.z < w.b.z)))) w.b = o;
            }
            far_settle(w, T, pix, site, sc, far, blockIdx.x);
        }
    }
    if (win_words && last_block(&ctr->ticket, gridDim.x)) decide_tile(bt, 0, sc, far, ctr, win_words);
}

// ---------------------------------------------------------------------------
// scatter-accumulate and finalize
// ---------------------------------------------------------------------------

__device__ __forceinline__ void emit_span(int row, int a, int b, int ncols, int nrows, bool packed,
                                          unsigned long long v, long long z,
                                          unsigned long long* __restrict__ D, int* __restrict__ Dc) {
    if (row < 0 || row >= nrows) return;
    a = a > 0 ? a : 0;
    b = b < ncols - 1 ? b : ncols - 1;
    if (a > b) return;
    const int64_t base = (int64_t)row * ncols;
    if (packed) {
        atomicAdd(&D[base + a], v);
        if (b + 1 < ncols) atomicAdd(&D[base + b + 1], (unsigned long long)(-(long long)v));
    } else {
        atomicAdd(&D[base + a], (unsigned long long)z);
        atomicAdd(&Dc[base + a], 1);
        if (b + 1 < ncols) {
            atomicAdd(&D[base + b + 1], (unsigned long long)(-z));
            atomicAdd(&Dc[base + b + 1], -1);
        }
    }
}

// The rows of one disc inside a chunk, walked from a per-lane start and
// wrapping at the last one: half_width() is floor(sqrt(R2 - dy^2)) of the
// current row, row its offset in the window.
//
// R2 < 2^20: t = R2 - dy^2 + 1/2 is exact in a float, and for k^2 <= t - 1/2 <
// (k+1)^2, k < 1024, its root lies at least 1/(4k+4) > 2.4e-4 from both k and
// k+1, twice the error of the hardware estimate (relative 2^-23, so 1.3e-4);
// the estimate rounded down is therefore the half-width itself (the tests run
// every value of the range on the device).  The floor
// is taken by adding 2^23 with rounding towards minus infinity, which leaves
// the integer in the low mantissa bits: no conversion instructions.  Larger
// discs take the estimate and one exact integer step each way.
struct SpanRows {
    float R2h, dyf, dy_last, back;
    int row, row_back, stride, R2;
    bool small;
    __device__ __forceinline__ SpanRows(int R2_, int dy, int dy_last_, int nrow, int row_, int stride_)
        : R2h((float)R2_ + 0.5f), dyf((float)dy), dy_last((float)dy_last_), back((float)(nrow - 1)), row(row_),
          row_back((nrow - 1) * stride_), stride(stride_), R2(R2_), small(R2_ < (1 << 20)) {}
    __device__ __forceinline__ int half_width() const {
        if (small) return __float_as_int(__fadd_rd(sqrt_est(fmaf(-dyf, dyf, R2h)), 8388608.0f)) - 0x4B000000;
        const int dy = (int)dyf;
        const unsigned t2 = (unsigned)R2 - (unsigned)(dy * dy);
        unsigned w = (unsigned)sqrt_est((float)t2);
        w -= (w * w > t2) ? 1u : 0u;
        w += ((w + 1) * (w + 1) <= t2) ? 1u : 0u;
        return (int)w;
    }
    __device__ __forceinline__ void next() {
        const bool wrap = dyf == dy_last;
        dyf = wrap ? dyf - back : dyf + 1.0f;
        row = wrap ? row - row_back : row + stride;
    }
};

// Span path: every pixel with R2 > rs^2 adds its disc as row spans (+v at
// the first cell, -v after the last, into the per-row difference words).
// Persistent CTAs (32 x 8 threads) take the work items of list_span_items:
// the rows of one group of chunks of one 32 x kTileY raster tile's window,
// whose chunks of whole rows fit `win_words` 8-byte cells of shared memory.
// For each chunk every disc of the tile adds its row spans' markers (z -
// zbase and 1 at the first cell, their negatives after the last) to two int32
// arrays with native shared-memory atomics, and each touched cell is then
// added to the grid's difference array as one packed word, (sum << K) +
// count, with one coalesced global atomic.  The markers of a tile's discs
// fall on far fewer distinct cells than there are markers (neighbouring
// pixels' discs share rows and end near each other), so the grid sees a
// fraction of the global atomics of the direct path, and those it sees are
// contiguous.  The sum is the same: the words add modulo 2^64 in any order
// and the packed form is linear.  Tiles with the unpacked accumulators
// (separate int64 Z and int32 C), with a z range the int32 window sums could
// overflow, or with windows wider than one chunk row, take the direct path.
//
// Bound by the shared-memory atomics' wavefronts (3.6 per instruction, banks
// hit at random): 76 % of the LSU's rate on the 4096^2, 20 M-point tile,
// 0.73 ms for its 3.7e8 span rows.  One CTA per raster tile took 1.75 ms (the
// lake tiles' CTAs ran alone on 46 % of the SM time), of it 0.3 ms for the
// conversions and correction steps of the half-widths; padding the window's
// row stride saved 5 % on 200 mixed tiles (1.23 -> 1.17 ms).
__global__ void __launch_bounds__(256) k_scatter_window(BatchTables bt, const int2* __restrict__ pix_all,
                                                        const Scalars* __restrict__ sc,
                                                        unsigned long long* __restrict__ D_all,
                                                        int* __restrict__ Dc_all, int win_words, FarLayout far,
                                                        BatchCounters* __restrict__ ctr, int nrt_layer,
                                                        int64_t lstride) {
    chained();
    extern __shared__ int swin[];              // 2 x win_words: z - zbase sums, then counts
    __shared__ int s_item;
    const int count = ctr->nspan;
    const int tid = threadIdx.y * 32 + threadIdx.x;
    const int ww4 = win_words & ~3;           // whole int4s
    int* sz = swin;                           // z - zbase sums
    int* scn = swin + ww4;                    // counts
    if (count > 0)                            // each chunk leaves the window zeroed
        for (int e = tid; e < ww4 >> 1; e += 256) reinterpret_cast<int4*>(swin)[e] = make_int4(0, 0, 0, 0);
    for (;;) {
    __syncthreads();                           // the previous item's reads of s_item are done
    if (tid == 0) s_item = atomicAdd(&ctr->span_next, 1);
    __syncthreads();
    if (s_item >= count) break;
    const int2 item = far.items[s_item];
    const int layer = nrt_layer ? item.x / nrt_layer : 0;
    const int rt = item.x - layer * nrt_layer;
    const int t = find_tile(bt.rt_base, bt.ntiles, rt);
    const TileParams T = bt.tiles[t];          // by value: the loops below keep what they use in registers
    const int2* pix = pix_all + T.pix_off + layer * lstride;
    const int lt = rt - __ldg(&bt.rt_base[t]);
    const int ntx = (T.rw + kTileX - 1) / kTileX;
    const int i = (lt % ntx) * kTileX + threadIdx.x;
    const int jt = (lt / ntx) * kTileY + threadIdx.y;
    const int rs2 = T.rs * T.rs;
    const int px = T.rx0 + i;
    const Scalars& s = sc[t];
    const bool direct = span_direct(s, s.bbox[4], s.bbox[5]);
    const SpanWindow win = span_window(T, lt, far.rtmax[item.x], win_words, direct);
    int R2v[kDenseSub], zv[kDenseSub], rv[kDenseSub];
#pragma unroll
    for (int sub = 0; sub < kDenseSub; ++sub) {
        const int j = jt + 8 * sub;
        int R2 = -1, z = 0;
        if (i < T.rw && j < T.rh) {
            const int2 r = pix[(int64_t)j * T.rw + i];
            z = r.x;
            R2 = r.y;
        }
        R2v[sub] = R2;
        zv[sub] = z;
        rv[sub] = R2 > rs2 ? isqrt_i32(R2) : -1;
    }
    unsigned long long* D = D_all + T.cell_off;
    int* Dc = Dc_all + T.cell_off;
    if (win.rows < 1) {
        // direct path: every span's markers straight to the grid
#pragma unroll 1
        for (int sub = 0; sub < kDenseSub; ++sub) {
            const int r = rv[sub];
            if (r < 0) continue;
            const int R2 = R2v[sub], z = zv[sub];
            const int py = T.ry0 + jt + 8 * sub;
            const unsigned long long v = span_word(z, s.zbase, s.kbits);
            int w = r;
            for (int dy = 0; dy <= r; ++dy) {
                const long long t2 = (long long)R2 - (long long)dy * dy;
                while ((long long)w * w > t2) --w;
                emit_span(py + dy, px - w, px + w, T.ncols, T.nrows, s.packed != 0, v, z, D, Dc);
                if (dy) emit_span(py - dy, px - w, px + w, T.ncols, T.nrows, s.packed != 0, v, z, D, Dc);
            }
        }
        continue;
    }
    const int W = win.W, SW = win.stride, CH = win.rows, c0 = win.c0;
    const int r0 = item.y, r1 = min(item.y + win.per - 1, win.r1);
    const bool inside = win.inside;
    const int ncols = T.ncols;
    const int zbase = (int)s.zbase;           // |z - zbase| fits (span_direct)
    const int kbits = s.kbits;
#pragma unroll 1
    for (int y0 = r0; y0 <= r1; y0 += CH) {
        const int y1 = min(y0 + CH - 1, r1);
#pragma unroll 1
        for (int sub = 0; sub < kDenseSub; ++sub) {
            const int r = rv[sub];
            if (r < 0) continue;
            const int py = T.ry0 + jt + 8 * sub;
            const int ya = max(py - r, y0), yb = min(py + r, y1);
            if (ya > yb) continue;
            const int zr = zv[sub] - zbase;
            // the lanes of a warp are 32 neighbouring pixels of one row, whose
            // markers on a common row often fall on one cell (same-address
            // atomics serialise); each lane starts its rows at its own offset
            // so that the warp's markers spread over the chunk's rows
            const int nrow = yb - ya + 1;
            const int y = ya + (int)(threadIdx.x % (unsigned)nrow);
            SpanRows rows(R2v[sub], y - py, yb - py, nrow, (y - y0) * SW - c0, SW);
            if (inside) {
#pragma unroll 2
                for (int k = 0; k < nrow; ++k) {
                    const int w = rows.half_width();
                    const int a = rows.row + px - w, b = rows.row + px + 1 + w;
                    atomicAdd(&sz[a], zr);
                    atomicAdd(&scn[a], 1);
                    atomicAdd(&sz[b], -zr);
                    atomicAdd(&scn[b], -1);
                    rows.next();
                }
            } else {
                for (int k = 0; k < nrow; ++k) {
                    const int w = rows.half_width();
                    const int a = max(px - w, 0), b = px + w + 1;
                    if (a < ncols && b > 0) {                // else this row's span misses the grid
                        atomicAdd(&sz[rows.row + a], zr);    // a and b lie in [c0, c1]
                        atomicAdd(&scn[rows.row + a], 1);
                        if (b < ncols) {
                            atomicAdd(&sz[rows.row + b], -zr);
                            atomicAdd(&scn[rows.row + b], -1);
                        }
                    }
                    rows.next();
                }
            }
        }
        __syncthreads();
        // one packed word per touched cell: (sum zrel << K) + count, modulo
        // 2^64; the cells read are zeroed for the next chunk
        for (int rr = threadIdx.y; rr <= y1 - y0; rr += 8) {
            unsigned long long* dst = D + (int64_t)(y0 + rr) * ncols + c0;
            for (int c = threadIdx.x; c < W; c += 32) {
                const int zs = sz[rr * SW + c], cn = scn[rr * SW + c];
                if (zs | cn) {
                    atomicAdd(&dst[c], ((unsigned long long)(long long)zs << kbits) + (unsigned long long)(long long)cn);
                    sz[rr * SW + c] = 0;
                    scn[rr * SW + c] = 0;
                }
            }
        }
        __syncthreads();
    }
    }
}

// Statistics only (not part of the launch sequence): spans per radius
// bucket of the span-path pixels (r = floor(sqrt(R2)), bucket = bit length
// of r), one CTA per 32 x kTileY raster tile.
__global__ void __launch_bounds__(256) k_span_hist(BatchTables bt, const int2* __restrict__ pix, Scalars* sc) {
    __shared__ unsigned hist[kSpanHistBuckets];
    const int tid = threadIdx.y * 32 + threadIdx.x;
    if (tid < kSpanHistBuckets) hist[tid] = 0;
    __syncthreads();
    const int t = find_tile(bt.rt_base, bt.ntiles, blockIdx.x);
    const TileParams& T = bt.tiles[t];
    const int lt = blockIdx.x - __ldg(&bt.rt_base[t]);
    const int ntx = (T.rw + kTileX - 1) / kTileX;
    const int i = (lt % ntx) * kTileX + threadIdx.x;
    const int rs2 = T.rs * T.rs;
    for (int sub = 0; sub < kDenseSub; ++sub) {
        const int j = (lt / ntx) * kTileY + threadIdx.y + 8 * sub;
        if (i >= T.rw || j >= T.rh) continue;
        const int R2 = pix[T.pix_off + (int64_t)j * T.rw + i].y;
        if (R2 <= rs2) continue;
        const int r = isqrt_i32(R2);
        const int k = min(32 - __clz(r), kSpanHistBuckets - 1);
        atomicAdd(&hist[k], 2u * (unsigned)r + 1u);
    }
    __syncthreads();
    if (tid < kSpanHistBuckets && hist[tid]) atomicAdd(&sc[t].span_hist[tid], (unsigned long long)hist[tid]);
}

// In-place inclusive prefix of one grid row (256 threads, 4 values each per step).
template <typename V>
__device__ __forceinline__ void row_prefix(V* __restrict__ row, int ncols, V* wsum) {
    V carry = 0;
    for (int base = 0; base < ncols; base += kScanThreads * 4) {
        const int idx = base + threadIdx.x * 4;
        V v[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) v[k] = (idx + k < ncols) ? row[idx + k] : V(0);
        v[1] += v[0]; v[2] += v[1]; v[3] += v[2];
        V total;
        const V excl = block_exclusive_sum(v[3], wsum, total, (int)threadIdx.x) + carry;
#pragma unroll
        for (int k = 0; k < 4; ++k) if (idx + k < ncols) row[idx + k] = v[k] + excl;
        carry += total;
    }
}

// One block per grid row: prefix of the span words, and of the int32 counts
// when the tile's accumulators are not packed.
__global__ void __launch_bounds__(kScanThreads) k_rowscan(BatchTables bt, unsigned long long* __restrict__ D_all,
                                                          int* __restrict__ Dc_all, const Scalars* __restrict__ sc) {
    __shared__ unsigned long long wsum[8];
    __shared__ int wsumc[8];
    const int t = find_tile(bt.grow_base, bt.ntiles, blockIdx.x);
    const TileParams& T = bt.tiles[t];
    const int64_t off = T.cell_off + (int64_t)(blockIdx.x - __ldg(&bt.grow_base[t])) * T.ncols;
    row_prefix(D_all + off, T.ncols, wsum);
    if (!sc[t].packed) row_prefix(Dc_all + off, T.ncols, wsumc);
}

__device__ __forceinline__ float finalize_height(long long Z, long long C, double zs, double zo, float nodata) {
    if (C <= 0) return nodata;
    const double q = __ddiv_rn(__ll2double_rn(Z), __ll2double_rn(C));
    return __double2float_rn(__dadd_rn(__dmul_rn(q, zs), zo));
}

// Lattice points within H of the origin.
constexpr int stencil_taps(int H) {
    int n = 0;
    for (int dy = -H; dy <= H; ++dy)
        for (int dx = -H; dx <= H; ++dx) n += dx * dx + dy * dy <= H * H ? 1 : 0;
    return n;
}

// Row scan, stencil and finalize in one pass: one CTA (32 x 16 threads) per
// band of 16 grid rows of a work package, walking the band's columns in
// chunks of 32.  Each warp owns one row: it prefix-sums the row's span words
// (the per-row difference form of the span path) chunk by chunk, carrying
// the running sum in a register, so the prefix is never written back; each
// cell then gathers the small discs (R2 <= H^2) of the pixels within H from
// the chunk's pixel records in shared memory, adds its prefix, and divides.
//
// A launch of fewer bands than SMs cuts them into segments of seg_cols columns,
// a CTA each (segs of them): a segment's rows start from the sum of the words
// before it, read once more.
//
// Bound by instruction issue (about 270 warp instructions per 32 cells, the
// double-precision quotient and the row scan more than the stencil) and the
// latency of the chunk chain.  512^2 cells (32 bands) 24.7 -> 12.0 us, mostly
// from sixteen segments; 1500 x 1400 cells 63.6 -> 45.2 us; 1024 mixed tiles 2.98 ->
// 2.61 ms from the chunk's record addresses formed once per band and stencil
// taps summed as one word.
template <int H>
__global__ void __launch_bounds__(512) k_rows_final(BatchTables bt, const int2* __restrict__ pix,
                                                    Scalars* __restrict__ sc,
                                                    const unsigned long long* __restrict__ S_all,
                                                    const int* __restrict__ Sc_all, float* __restrict__ h_all, int segs,
                                                    int seg_cols) {
    chained();
    constexpr int TX = 32, TY = 16, SW = TX + 2 * H, SH = TY + 2 * H;
    constexpr int NL = (SW * SH + TX * TY - 1) / (TX * TY);   // pixel records each thread loads per chunk
    __shared__ int2 tile[2][SH][SW];                          // double buffer: this chunk and the next
    const int band = blockIdx.x / segs, c_begin = (blockIdx.x - band * segs) * seg_cols;
    const int t = find_tile(bt.band_base, bt.ntiles, band);
    const TileParams T = bt.tiles[t];
    if (c_begin >= T.ncols) return;
    const int c_end = min(c_begin + seg_cols, T.ncols);
    const int cy0 = (band - __ldg(&bt.band_base[t])) * TY;
    const int2* P = pix + T.pix_off;
    Scalars* s = sc + t;
    const bool packed = s->packed != 0;
    const int K = s->kbits;
    const long long zbase = s->zbase;
    // a record's place in the stencil: (z - zbase) * 2^KB + 1 and its R2, -1
    // when the span path has it, so that a cell sums its taps' values and counts
    // in one 32-bit word; where the sum could overflow (`wide`), z itself
    constexpr int TAPS = stencil_taps(H), KB = TAPS < 32 ? 5 : (TAPS < 64 ? 6 : 7);
    const long long zabs = max((long long)s->bbox[5] - zbase, zbase - (long long)s->bbox[4]);
    const bool wide = zabs >= (1LL << (31 - KB)) / (TAPS + 1);
    const int zb32 = (int)zbase;
    const int lane = threadIdx.x, tid = threadIdx.y * TX + threadIdx.x;
    const int qy = cy0 + threadIdx.y;
    const bool row_in = qy < T.nrows;
    // the chunk starting at column cx: this thread's pixel records (into
    // registers) and its cell's span words
    int2 rec[NL];
    const int2* src[NL];                 // the record at column cx = 0, its raster column there, its place in a buffer
    int col[NL], at[NL];
#pragma unroll
    for (int k = 0; k < NL; ++k) {
        const int idx = tid + k * TX * TY, ly = idx / SW, lx = idx - ly * SW;
        const int ryi = cy0 - H + ly - T.ry0;
        at[k] = idx;
        col[k] = idx < SW * SH && ryi >= 0 && ryi < T.rh ? lx - H - T.rx0 : INT_MIN / 2;   // never inside
        src[k] = P + ((int64_t)ryi * T.rw + col[k]);
    }
    auto load_tile = [&](int cx) {
#pragma unroll
        for (int k = 0; k < NL; ++k) {
            int2 v = make_int2(0, -1);
            if ((unsigned)(col[k] + cx) < (unsigned)T.rw) v = src[k][cx];
            rec[k] = v;
        }
    };
    auto store_tile = [&](int b) {
#pragma unroll
        for (int k = 0; k < NL; ++k) {
            int2 v = rec[k];
            if (v.y > H * H) v.y = -1;
            if (!wide) v.x = (v.x - zb32) * (1 << KB) + 1;
            if (k < NL - 1 || at[k] < SW * SH) (&tile[b][0][0])[at[k]] = v;
        }
    };
    auto load_words = [&](int cx, unsigned long long& w, int& wc) {
        const int qx = cx + lane;
        const bool in = row_in && qx < T.ncols;
        const int64_t q = (int64_t)qy * T.ncols + qx;
        w = in ? S_all[T.cell_off + q] : 0ull;
        wc = (in && !packed) ? Sc_all[T.cell_off + q] : 0;
    };
    unsigned long long carry = 0;   // running prefix of the row's span words (Z when unpacked)
    int carry_c = 0;                // running prefix of the counts (unpacked)
    unsigned nod = 0;
    unsigned long long w;
    int wc;
    load_tile(c_begin);
    store_tile(0);
    load_words(c_begin, w, wc);
    if (c_begin > 0 && row_in) {
        // the words before this segment
        const int64_t q = T.cell_off + (int64_t)qy * T.ncols;
#pragma unroll 4
        for (int c = lane; c < c_begin; c += TX) {
            carry += S_all[q + c];
            if (!packed) carry_c += Sc_all[q + c];
        }
#pragma unroll
        for (int o = 16; o; o >>= 1) {
            carry += __shfl_xor_sync(0xffffffffu, carry, o);
            carry_c += __shfl_xor_sync(0xffffffffu, carry_c, o);
        }
    }
    __syncthreads();
    int b = 0;
#pragma unroll 1
    for (int cx0 = c_begin; cx0 < c_end; cx0 += TX, b ^= 1) {
        // the next chunk's loads are in flight while this one computes
        const bool more = cx0 + TX < c_end;
        unsigned long long w_next = 0;
        int wc_next = 0;
        if (more) {
            load_tile(cx0 + TX);
            load_words(cx0 + TX, w_next, wc_next);
        }
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned long long y = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) w += y;
        }
        w += carry;
        carry = __shfl_sync(0xffffffffu, w, 31);
        if (!packed) {
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int yc = __shfl_up_sync(0xffffffffu, wc, o);
                if (lane >= o) wc += yc;
            }
            wc += carry_c;
            carry_c = __shfl_sync(0xffffffffu, wc, 31);
        }
        long long Z = 0, C = 0;
        if (!wide) {
            int sum = 0;
#pragma unroll
            for (int dy = -H; dy <= H; ++dy)
#pragma unroll
                for (int dx = -H; dx <= H; ++dx) {
                    if (dx * dx + dy * dy > H * H) continue;
                    const int2 p = tile[b][threadIdx.y + H + dy][lane + H + dx];
                    if (p.y >= dx * dx + dy * dy) sum += p.x;
                }
            C = sum & ((1 << KB) - 1);
            Z = (long long)(sum >> KB) + C * zbase;
        } else {
#pragma unroll 1
            for (int dy = -H; dy <= H; ++dy)
#pragma unroll 1
                for (int dx = -H; dx <= H; ++dx) {
                    const int d2 = dx * dx + dy * dy;
                    const int2 p = tile[b][threadIdx.y + H + dy][lane + H + dx];
                    if (d2 <= H * H && p.y >= d2) { Z += p.x; C += 1; }
                }
        }
        const int qx = cx0 + lane;
        if (row_in && qx < T.ncols) {
            if (packed) {
                long long zb, cb;
                decode_span_word(w, K, zbase, zb, cb);
                Z += zb;
                C += cb;
            } else {
                Z += (long long)w;
                C += wc;
            }
            h_all[T.out_off + (int64_t)qy * T.ncols + qx] = finalize_height(Z, C, T.z_scale, T.z_offset, T.nodata);
            nod += C <= 0 ? 1u : 0u;
        }
        if (more) {
            // the other buffer's last readers (the chunk before this one)
            // finished before the barrier that ended that chunk
            store_tile(b ^ 1);
            w = w_next;
            wc = wc_next;
        }
        __syncthreads();
    }
    nod = __reduce_add_sync(0xffffffffu, nod);
    if (lane == 0 && nod) {
        const int slot = (blockIdx.x + threadIdx.y) & (kStatSlots - 1);
        atomicAdd(&s->nodata[slot], (unsigned long long)nod);
    }
}

}  // namespace dnni
