// dnni_compat.cuh -- the reference's own default semantics on the GPU
// (dnni_interpolate_compat): square site regions, a pixel lattice `scale`
// times finer than the cells, float32 lifted-plane depths with the
// later-drawn site winning equal depths, square query regions, int32 z-codes
// summed with wrap-around and a truncating divide.  Included by
// dnni_engine.cu.
//
// Follows nni::performNNI for timeRadius == 0 with the plane algorithm:
//   pixel_offset and raster size                   nni.cpp:879-886
//   site squares, z-code, depth test (LEQUAL)      nni.cpp:171-230, 470-479, 538-549, 733-737
//   query squares tested against the stored depth  nni.cpp:483-534, 803-807
//   int32 numer/denom, truncating divide           cuda_nni.cu:423-448, 491-503
//   dequantisation                                 nni.cpp:836-848
// evaluating each plane at pixel centres over the half-open square
// [x - r, x + r) x [y - r, y + r); the GL rasteriser's fill rule and its
// depth interpolation are not reproduced.  Every floating-point operation is
// written with an explicit rounding intrinsic, in the order the formulas
// give, so that no multiply-add is fused and the results are those of the
// same formulas evaluated in IEEE single and double precision on the host.
#pragma once

namespace dnni {

struct CompatGeom {
    double pixel_size, left, bottom, rs, rq, qspacing;
    float hw;
    int32_t xp, yp, ncols, nrows, z_offset, z_mult;
    float ox, oy;
};

// A site's (or query's) lifted plane: its slopes and offset depend on the
// point only, so they are formed once per point, as drawPlane forms them
// (nni.cpp:186-200): the point's offset (dx, dy) from the work-package
// origin stays in double, zpx = (dx + halfwidth) / halfwidth and the slopes
// a = -2.0 * zpx / halfwidth are evaluated in double and rounded to float
// once each, and the offset is the float sum of the float squares (the time
// term is zero in 2-D).
struct CompatPlane {
    float a, b, zoff;
};

__device__ __forceinline__ CompatPlane compat_plane(float hw, double dx, double dy) {
    const double h = (double)hw;
    const float zpx = __double2float_rn(__ddiv_rn(__dadd_rn(dx, h), h));
    const float zpy = __double2float_rn(__ddiv_rn(__dadd_rn(dy, h), h));
    CompatPlane P;
    P.zoff = __fadd_rn(__fmul_rn(zpx, zpx), __fmul_rn(zpy, zpy));
    P.a = __double2float_rn(__ddiv_rn(__dmul_rn(-2.0, (double)zpx), h));
    P.b = __double2float_rn(__ddiv_rn(__dmul_rn(-2.0, (double)zpy), h));
    return P;
}

// The plane's depth at a pixel centre (px, py).
__device__ __forceinline__ float compat_depth(const CompatPlane& P, float hw, float px, float py) {
    const float zx = __fadd_rn(px, hw), zy = __fadd_rn(py, hw);
    return __fadd_rn(__fadd_rn(__fmul_rn(P.a, zx), __fmul_rn(P.b, zy)), P.zoff);
}

// Pixel index range [i0, i1] whose centres fall in [x0, x1) (one axis).
__device__ __forceinline__ void compat_span(float x0, float x1, double left, double ps, long long n, long long& i0,
                                            long long& i1) {
    i0 = (long long)ceil(__dsub_rn(__ddiv_rn(__dsub_rn((double)x0, left), ps), 0.5));
    i1 = (long long)ceil(__dsub_rn(__ddiv_rn(__dsub_rn((double)x1, left), ps), 0.5)) - 1;
    if (i0 < 0) i0 = 0;
    if (i1 > n - 1) i1 = n - 1;
}

__device__ __forceinline__ float compat_centre(long long p, double base, double ps) {
    return __double2float_rn(__dadd_rn(base, __dmul_rn((double)p + 0.5, ps)));
}

// Order-preserving map of a float's bits to an unsigned integer.
__device__ __forceinline__ uint32_t compat_order(float d) {
    const uint32_t u = __float_as_uint(d);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float compat_unorder(uint32_t o) {
    return __uint_as_float((o & 0x80000000u) ? (o & 0x7FFFFFFFu) : ~o);
}

// A point's square of site influence: its offset from the work package
// (double, and rounded to float as drawPlane's px, py) and the pixels
// [i0,i1] x [j0,j1] whose centres the square covers (empty when i0 > i1 or
// j0 > j1).
struct CompatSquare {
    double dx, dy;
    float sx, sy;
    long long i0, i1, j0, j1;
};

__device__ __forceinline__ CompatSquare compat_square(const CompatGeom& G, const double* __restrict__ xyz, int64_t k) {
    CompatSquare q;
    q.dx = __dsub_rn(xyz[3 * k], (double)G.ox);
    q.dy = __dsub_rn(xyz[3 * k + 1], (double)G.oy);
    q.sx = __double2float_rn(q.dx);
    q.sy = __double2float_rn(q.dy);
    const float x0 = __double2float_rn(__dsub_rn((double)q.sx, G.rs)), x1 = __double2float_rn(__dadd_rn((double)q.sx, G.rs));
    const float y0 = __double2float_rn(__dsub_rn((double)q.sy, G.rs)), y1 = __double2float_rn(__dadd_rn((double)q.sy, G.rs));
    compat_span(x0, x1, G.left, G.pixel_size, G.xp, q.i0, q.i1);
    compat_span(y0, y1, G.bottom, G.pixel_size, G.yp, q.j0, q.j1);
    return q;
}

// z-code of a point: floor((z + zOffset + 1) * zMult) (nni.cpp:538-549).
__device__ __forceinline__ uint32_t compat_zcode(double z, int z_offset, int z_mult) {
    return (uint32_t)(long long)floor(__dmul_rn(__dadd_rn(__dadd_rn(z, (double)z_offset), 1.0), (double)z_mult));
}

// A pixel as the query pass reads it: the depth of the site it kept (as
// compat_order gives it) and that site's z-code, 0 when it counts for no cell
// (no site, or a site whose code is zero).
__device__ __forceinline__ uint2 compat_pixel(const CompatGeom& G, const double* __restrict__ xyz,
                                              unsigned long long key) {
    if (key == ~0ull) return make_uint2(0xFFFFFFFFu, 0u);
    const int64_t k = (int64_t)(0xFFFFFFFFull - (key & 0xFFFFFFFFull));
    return make_uint2((uint32_t)(key >> 32), compat_zcode(xyz[3 * k + 2], G.z_offset, G.z_mult));
}

// ---- site pass by gather ----
//
// Each point is filed once, under the raster tile of kCgTile x kCgTile pixels
// that holds the first pixel of its square, as a record of its plane, draw order
// and square (k_cg_count, k_cg_offsets, k_cg_fill).  A square reaches at most
// `reach` tiles to the right and up, so a tile's points are `reach` + 1 ranges of
// records, one per row of home tiles.  One CTA per tile loads them, keeps those
// that meet the tile, and each warp runs over the ones that meet its 8 x 4
// pixels, every lane keeping its pixel's least key in registers.
//
// Bound by instruction issue (79 % of the slots: plane, key and comparison of
// about 89 candidates per pixel at 1 point per m^2, of which 50 cover it; the
// squares' bounds are tested once per point, as a mask of the lanes they cover).
// 3.6 M points on 1000 x 900 cells at 5 pixels per cell: 1.81 ms (filing 0.20
// ms); taking each covered pixel's minimum with a 64-bit shared-memory atomic, a
// compare-and-swap loop each, 5.94 ms (filing 0.56 ms).
constexpr int kCgTile = 32;
constexpr int kCgRound = 512;               // source points per round of a CTA

struct CgRecs {
    float4* plane;                          // a, b, zoff, the key's low word (bits)
    uint2* box;                             // i0 | j0 << 16, i1 | j1 << 16
};

__global__ void __launch_bounds__(256) k_cg_count(CompatGeom G, const double* __restrict__ xyz, int64_t n, int ntx,
                                                  int* __restrict__ tcnt) {
    const int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (k >= n) return;
    const CompatSquare q = compat_square(G, xyz, k);
    if (q.i0 > q.i1 || q.j0 > q.j1) return;
    atomicAdd(&tcnt[(q.j0 / kCgTile) * ntx + q.i0 / kCgTile], 1);
}

// One CTA: exclusive prefix of the nt tile counts into toff[0..nt]; the counts
// become fill cursors at zero.
__global__ void __launch_bounds__(1024) k_cg_offsets(int* __restrict__ tcnt, int nt, long long* __restrict__ toff) {
    __shared__ long long wsum[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    long long carry = 0;
    for (int b = 0; b < nt; b += 4096) {
        const int k0 = b + 4 * threadIdx.x;
        int v[4];
        long long s = 0;
#pragma unroll
        for (int k = 0; k < 4; ++k) { v[k] = k0 + k < nt ? tcnt[k0 + k] : 0; s += v[k]; }
        long long x = s;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) { const long long y = __shfl_up_sync(0xffffffffu, x, o); if (lane >= o) x += y; }
        if (lane == 31) wsum[warp] = x;
        __syncthreads();
        long long w = wsum[lane];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) { const long long y = __shfl_up_sync(0xffffffffu, w, o); if (lane >= o) w += y; }
        const long long before = __shfl_sync(0xffffffffu, w, (warp + 31) & 31), total = __shfl_sync(0xffffffffu, w, 31);
        long long run = carry + x - s + (warp ? before : 0);
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (k0 + k < nt) { toff[k0 + k] = run; run += v[k]; tcnt[k0 + k] = 0; }
        carry += total;
        __syncthreads();
    }
    if (threadIdx.x == 0) toff[nt] = carry;
}

__global__ void __launch_bounds__(256) k_cg_fill(CompatGeom G, const double* __restrict__ xyz, int64_t n, int ntx,
                                                 const long long* __restrict__ toff, int* __restrict__ tcur, CgRecs R) {
    const int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (k >= n) return;
    const CompatSquare q = compat_square(G, xyz, k);
    if (q.i0 > q.i1 || q.j0 > q.j1) return;
    const long long t = (q.j0 / kCgTile) * ntx + q.i0 / kCgTile;
    const long long e = toff[t] + atomicAdd(&tcur[t], 1);
    const CompatPlane P = compat_plane(G.hw, q.dx, q.dy);
    R.plane[e] = make_float4(P.a, P.b, P.zoff, __uint_as_float(0xFFFFFFFFu - (uint32_t)k));
    R.box[e] = make_uint2((uint32_t)q.i0 | (uint32_t)q.j0 << 16, (uint32_t)q.i1 | (uint32_t)q.j1 << 16);
}

__global__ void __launch_bounds__(256) k_cg_sites(CompatGeom G, const double* __restrict__ xyz, int ntx, int reach,
                                                  const long long* __restrict__ toff, CgRecs R,
                                                  uint2* __restrict__ pixel) {
    __shared__ float4 s_plane[kCgRound];
    __shared__ int4 s_box[kCgRound];        // i0, i1, j0, j1
    __shared__ unsigned short s_list[8][kCgRound];
    __shared__ unsigned s_mask[8][kCgRound];
    __shared__ int s_n;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const unsigned own = 1u << lane, below = own - 1u;
    const int tx = blockIdx.x % ntx, ty = blockIdx.x / ntx;
    const int px0 = tx * kCgTile, py0 = ty * kCgTile;
    // a warp's strip of four rows, an 8 x 4 block of it at a time; this lane's
    // pixels and their lattice coordinates
    const int pj = py0 + 4 * warp + (lane >> 3), y0 = py0 + 4 * warp;
    const float zy = __fadd_rn(compat_centre(pj, G.bottom, G.pixel_size), G.hw);
    float zx[4];
    unsigned long long best[4];             // least key, all ones: none
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        zx[c] = __fadd_rn(compat_centre(px0 + 8 * c + (lane & 7), G.left, G.pixel_size), G.hw);
        best[c] = ~0ull;
    }
    unsigned short* list = s_list[warp];
    unsigned* mask = s_mask[warp];
    for (int hy = max(ty - reach, 0); hy <= ty; ++hy) {
        const long long e0 = toff[(long long)hy * ntx + max(tx - reach, 0)], e1 = toff[(long long)hy * ntx + tx + 1];
        for (long long b = e0; b < e1; b += kCgRound) {
            __syncthreads();                // the previous round's readers are done
            if (tid == 0) s_n = 0;
            __syncthreads();
            const int m = (int)min((long long)kCgRound, e1 - b);
            for (int q0 = 0; q0 < m; q0 += 256) {
                const int q = q0 + tid;
                bool in = false;
                uint2 box = make_uint2(0, 0);
                if (q < m) {
                    box = R.box[b + q];
                    in = (int)(box.y & 0xFFFF) >= px0 && (int)(box.y >> 16) >= py0;
                }
                const unsigned got = __ballot_sync(0xffffffffu, in);
                int base = 0;
                if (lane == 0 && got) base = atomicAdd(&s_n, __popc(got));
                base = __shfl_sync(0xffffffffu, base, 0) + __popc(got & below);
                if (in) {
                    s_plane[base] = R.plane[b + q];
                    s_box[base] = make_int4(box.x & 0xFFFF, box.y & 0xFFFF, box.x >> 16, box.y >> 16);
                }
            }
            __syncthreads();
            const int n = s_n;
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                // the points that meet these 8 x 4 pixels, with the lanes
                // (row-major) whose pixels each one's square covers
                const int x0 = px0 + 8 * c;
                int cnt = 0;
                for (int q0 = 0; q0 < n; q0 += 32) {
                    const int q = q0 + lane;
                    unsigned cover = 0;
                    if (q < n) {
                        const int4 v = s_box[q];
                        const int a0 = max(v.x - x0, 0), a1 = min(v.y - x0, 7), b0 = max(v.z - y0, 0), b1 = min(v.w - y0, 3);
                        if (a0 <= a1 && b0 <= b1)
                            cover = (((0xFFu >> (7 - a1 + a0)) << a0) * 0x01010101u) & (0xFFFFFFFFu << (8 * b0)) &
                                    (0xFFFFFFFFu >> (8 * (3 - b1)));
                    }
                    const unsigned got = __ballot_sync(0xffffffffu, cover != 0);
                    if (cover) {
                        const int e = cnt + __popc(got & below);
                        list[e] = (unsigned short)q;
                        mask[e] = cover;
                    }
                    cnt += __popc(got);
                }
                __syncwarp();
                unsigned long long bc = best[c];
#pragma unroll 4
                for (int q = 0; q < cnt; ++q) {
                    const float4 P = s_plane[list[q]];
                    const float d = __fadd_rn(__fadd_rn(__fmul_rn(P.x, zx[c]), __fmul_rn(P.y, zy)), P.z);
                    const unsigned long long key = ((unsigned long long)compat_order(d) << 32) | __float_as_uint(P.w);
                    const bool less = (mask[q] & own) && key < bc;
                    bc = less ? key : bc;
                }
                best[c] = bc;
                __syncwarp();
            }
        }
    }
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        const int pi = px0 + 8 * c + (lane & 7);
        if (pi < G.xp && pj < G.yp) pixel[(long long)pj * G.xp + pi] = compat_pixel(G, xyz, best[c]);
    }
}

// ---- site pass by shared-memory minima: for callers whose scratch limit
// leaves no room for the records ----
//
// It runs per raster tile of kCpTile x kCpTile pixels whose keys
// sit in shared memory: the points are first listed per tile they reach
// (k_compat_count, k_compat_offsets, k_compat_fill), then one CTA per tile
// takes the minimum key of its points per pixel and writes the tile out once.
constexpr int kCpTile = 96;
constexpr size_t kCpTileSmem = sizeof(unsigned long long) * kCpTile * kCpTile;

__global__ void __launch_bounds__(256) k_compat_count(CompatGeom G, const double* __restrict__ xyz, int64_t n,
                                                      int ntx, int* __restrict__ tcnt) {
    for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < n; k += (int64_t)gridDim.x * blockDim.x) {
        const CompatSquare q = compat_square(G, xyz, k);
        if (q.i0 > q.i1 || q.j0 > q.j1) continue;
        for (long long ty = q.j0 / kCpTile; ty <= q.j1 / kCpTile; ++ty)
            for (long long tx = q.i0 / kCpTile; tx <= q.i1 / kCpTile; ++tx) atomicAdd(&tcnt[ty * ntx + tx], 1);
    }
}

// One CTA of 1024 threads: exclusive prefix of the nt tile counts into
// toff[0..nt] and zeroed fill cursors.
__global__ void __launch_bounds__(1024) k_compat_offsets(const int* __restrict__ tcnt, int nt, long long* __restrict__ toff,
                                                         int* __restrict__ tcur) {
    __shared__ long long wsum[32];
    const int per = (nt + 1023) / 1024;
    const int b0 = threadIdx.x * per;
    long long s = 0;
    for (int k = 0; k < per; ++k) if (b0 + k < nt) s += tcnt[b0 + k];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    long long x = s;
    for (int o = 1; o < 32; o <<= 1) { const long long y = __shfl_up_sync(0xffffffffu, x, o); if (lane >= o) x += y; }
    if (lane == 31) wsum[warp] = x;
    __syncthreads();
    if (warp == 0) {
        long long w = wsum[lane];
        for (int o = 1; o < 32; o <<= 1) { const long long y = __shfl_up_sync(0xffffffffu, w, o); if (lane >= o) w += y; }
        wsum[lane] = w;
    }
    __syncthreads();
    long long run = x - s + (warp ? wsum[warp - 1] : 0);
    for (int k = 0; k < per; ++k)
        if (b0 + k < nt) { toff[b0 + k] = run; run += tcnt[b0 + k]; tcur[b0 + k] = 0; }
    if (threadIdx.x == 1023) toff[nt] = run;
}

// (cap: the list's capacity, a bound on the squares' tile counts that the
// host derives from the site radius; entries past it are dropped, never written)
__global__ void __launch_bounds__(256) k_compat_fill(CompatGeom G, const double* __restrict__ xyz, int64_t n, int ntx,
                                                     const long long* __restrict__ toff, int* __restrict__ tcur,
                                                     uint32_t* __restrict__ list, int64_t cap) {
    for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < n; k += (int64_t)gridDim.x * blockDim.x) {
        const CompatSquare q = compat_square(G, xyz, k);
        if (q.i0 > q.i1 || q.j0 > q.j1) continue;
        for (long long ty = q.j0 / kCpTile; ty <= q.j1 / kCpTile; ++ty)
            for (long long tx = q.i0 / kCpTile; tx <= q.i1 / kCpTile; ++tx) {
                const long long t = ty * ntx + tx;
                const long long e = toff[t] + atomicAdd(&tcur[t], 1);
                if (e < cap) list[e] = (uint32_t)k;
            }
    }
}

// Site pass, one CTA per tile: every pixel keeps the smallest depth of the
// points whose squares cover it, the largest draw order k among equal depths
// (the depth test's later-draw-wins), as the 64-bit key order(d) << 32 | ~k;
// ~0 where no square reaches.
__global__ void __launch_bounds__(256) k_compat_sites(CompatGeom G, const double* __restrict__ xyz, int ntx,
                                                      const long long* __restrict__ toff,
                                                      const uint32_t* __restrict__ list, int64_t cap,
                                                      uint2* __restrict__ pixel) {
    extern __shared__ unsigned long long sk[];
    const int t = blockIdx.x;
    const long long px0 = (long long)(t % ntx) * kCpTile, py0 = (long long)(t / ntx) * kCpTile;
    const int pw = (int)min((long long)kCpTile, (long long)G.xp - px0);
    const int ph = (int)min((long long)kCpTile, (long long)G.yp - py0);
    for (int e = threadIdx.x; e < kCpTile * kCpTile; e += blockDim.x) sk[e] = ~0ull;
    __syncthreads();
    const long long e1 = toff[t + 1] < cap ? toff[t + 1] : (long long)cap;
    for (long long e = toff[t] + threadIdx.x; e < e1; e += blockDim.x) {
        const int64_t k = list[e];
        const CompatSquare q = compat_square(G, xyz, k);
        const long long i0 = max(q.i0, px0), i1 = min(q.i1, px0 + pw - 1);
        const long long j0 = max(q.j0, py0), j1 = min(q.j1, py0 + ph - 1);
        const unsigned long long low = 0xFFFFFFFFull - (unsigned long long)k;
        const CompatPlane P = compat_plane(G.hw, q.dx, q.dy);
        for (long long pj = j0; pj <= j1; ++pj) {
            const float cy = compat_centre(pj, G.bottom, G.pixel_size);
            for (long long pi = i0; pi <= i1; ++pi) {
                const float cx = compat_centre(pi, G.left, G.pixel_size);
                const float d = compat_depth(P, G.hw, cx, cy);
                atomicMin(&sk[(pj - py0) * kCpTile + (pi - px0)], ((unsigned long long)compat_order(d) << 32) | low);
            }
        }
    }
    __syncthreads();
    for (int e = threadIdx.x; e < kCpTile * kCpTile; e += blockDim.x) {
        const int r = e / kCpTile, c = e - r * kCpTile;
        if (r < ph && c < pw) pixel[(py0 + r) * G.xp + px0 + c] = compat_pixel(G, xyz, sk[e]);
    }
}

// (The pixels hold their sites' z-codes: looking each up through its point, per
// cell and pixel, took 0.80 ms where this takes 0.30 ms.)
// Query pass and divide: one thread per cell, over the pixels of its square;
// a pixel counts when it holds a site with a non-zero z-code and the cell's
// own plane is no deeper there (cuda_nni.cu:423-448).
__global__ void __launch_bounds__(256) k_compat_cells(CompatGeom G, const uint2* __restrict__ pixel,
                                                      float* __restrict__ h, int32_t* __restrict__ res) {
    const int64_t w = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (w >= (int64_t)G.ncols * G.nrows) return;
    const int i = (int)(w % G.ncols), j = (int)(w / G.ncols);
    const double qdx = __dmul_rn((double)i, G.qspacing), qdy = __dmul_rn((double)j, G.qspacing);
    const float qx = __double2float_rn(qdx);
    const float qy = __double2float_rn(qdy);
    const float x0 = __double2float_rn(__dsub_rn((double)qx, G.rq)), x1 = __double2float_rn(__dadd_rn((double)qx, G.rq));
    const float y0 = __double2float_rn(__dsub_rn((double)qy, G.rq)), y1 = __double2float_rn(__dadd_rn((double)qy, G.rq));
    long long i0, i1, j0, j1;
    compat_span(x0, x1, G.left, G.pixel_size, G.xp, i0, i1);
    compat_span(y0, y1, G.bottom, G.pixel_size, G.yp, j0, j1);
    uint32_t numer = 0;
    int32_t denom = 0;
    const CompatPlane Q = compat_plane(G.hw, qdx, qdy);
    for (int pj = (int)j0; pj <= (int)j1; ++pj) {
        const float zb = __fmul_rn(Q.b, __fadd_rn(compat_centre(pj, G.bottom, G.pixel_size), G.hw));
        const uint2* row = pixel + (long long)pj * G.xp;
#pragma unroll 4
        for (int pi = (int)i0; pi <= (int)i1; ++pi) {
            const uint2 p = __ldg(&row[pi]);
            const float za = __fmul_rn(Q.a, __fadd_rn(compat_centre(pi, G.left, G.pixel_size), G.hw));
            const float d = __fadd_rn(__fadd_rn(za, zb), Q.zoff);
            if (p.y != 0 && d <= compat_unorder(p.x)) {
                numer += p.y;                                 // int32 sum with wrap, as the atomicAdd
                denom += 1;
            }
        }
    }
    const int32_t r = denom == 0 ? -9999 * G.z_mult : (int32_t)numer / denom;
    if (res) res[w] = r;
    double z = __ddiv_rn((double)r, (double)G.z_mult);
    if (z != -9999.0) z = __dsub_rn(__dsub_rn(z, (double)G.z_offset), 1.0);
    h[w] = __double2float_rn(z);
}

}  // namespace dnni

// Both entry points: host buffers (device = false: points copied in,
// heights and quotients copied out, the call waits) or device buffers
// (queued on st; the call returns with the work queued).
static dnni_status compat_run(dnni_ctx* c, const dnni_compat_settings* s, const dnni_compat_wp* wp, const double* xyz,
                              int64_t n, float* h_out, int32_t* res_out, bool device, cudaStream_t st) {
    if (s->scale <= 0 || !(s->cell_size > 0) || wp->nrows <= 0 || wp->ncols <= 0 || s->multiplier <= 0)
        return set_err(c, DNNI_E_INVAL, "scale, cell size, grid sides and multiplier must be positive");
    if ((uint64_t)n >= 0xFFFFFFFFull) return set_err(c, DNNI_E_INVAL, "too many points for 32-bit draw order");
    // geometry as nni::performNNI derives it (nni.cpp:879-886, 186-189)
    CompatGeom G;
    G.qspacing = s->cell_size;
    G.pixel_size = G.qspacing / s->scale;
    const float qr = (float)s->query_radius;
    const int pixel_offset = (int)std::ceil((qr - std::floor(s->scale / 2.0) * G.pixel_size) / G.pixel_size) + 1;
    const long long xp = (long long)wp->ncols * s->scale + 2LL * pixel_offset;
    const long long yp = (long long)wp->nrows * s->scale + 2LL * pixel_offset;
    if (xp <= 0 || yp <= 0 || xp > 65535 || yp > 65535 || xp * yp > (1LL << 31))
        return set_err(c, DNNI_E_INVAL, "raster of the work package too large");
    G.xp = (int32_t)xp;
    G.yp = (int32_t)yp;
    G.left = 0 - (G.qspacing / 2.0) - (pixel_offset * G.pixel_size);
    G.bottom = G.left;
    G.hw = (float)(((wp->nrows - 1) * G.qspacing) / 2.0);
    G.rs = s->site_radius / std::sqrt(2.0);
    G.rq = qr / std::sqrt(2.0);
    G.ncols = wp->ncols;
    G.nrows = wp->nrows;
    G.z_offset = -1 * s->point_min;
    G.z_mult = s->multiplier;
    G.ox = wp->origin_x;
    G.oy = wp->origin_y;
    const int64_t cells = (int64_t)wp->ncols * wp->nrows;
    // scratch: the pixels in the context's late buffer; the gather's tile offsets,
    // counts (or cursors) and records in its optional buffer, or else the tile
    // counts, offsets and cursors in its bin-count buffer and the per-tile point
    // lists in its list buffer; points and outputs in its staging buffers
    dnni_status rs;
    if ((rs = dnni_ensure(c, c->scr.late, sizeof(uint2) * (size_t)(xp * yp))) ||
        (!device && ((rs = dnni_ensure(c, c->in_xyz, sizeof(double) * 3 * (size_t)std::max<int64_t>(n, 1))) ||
                     (rs = dnni_ensure(c, c->out_h, sizeof(float) * (size_t)cells)) ||
                     (res_out && (rs = dnni_ensure(c, c->out_site, sizeof(int32_t) * (size_t)cells))))))
        return rs;
    const double* dxyz = device ? xyz : (const double*)c->in_xyz.p;
    float* dh = device ? h_out : (float*)c->out_h.p;
    int32_t* dres = res_out ? (device ? res_out : (int32_t*)c->out_site.p) : nullptr;
    uint2* pixel = (uint2*)c->scr.late.p;
    // pixels of the raster that one square spans at most, one axis (with its rounding)
    const double across = std::ceil(2.0 * G.rs / G.pixel_size), most = (double)std::max(xp, yp);
    const long long span = (long long)(across < most ? across : most) + 3;
    // the offsets, then the counts, of nt tiles
    auto tile_bytes = [](long long nt, int per_tile) { return sizeof(long long) * (size_t)(nt + 1) + per_tile * sizeof(int) * (size_t)nt; };
    const long long gx = (xp + kCgTile - 1) / kCgTile, gy = (yp + kCgTile - 1) / kCgTile;
    const size_t recs = (size_t)std::max<int64_t>(n, 1), tiles = al256(tile_bytes(gx * gy, 1));
    void* gather = ensure_optional(c, c->scr.part, tiles + (sizeof(float4) + sizeof(uint2)) * recs);
    if (gather) {
        const int nt = (int)(gx * gy);
        long long* toff = (long long*)gather;
        int* tcnt = (int*)(toff + nt + 1);
        float4* plane = (float4*)((unsigned char*)gather + tiles);
        const CgRecs R{plane, (uint2*)(plane + recs)};
        const unsigned blocks = (unsigned)((n + 255) / 256);
        CK(cudaMemsetAsync(tcnt, 0, sizeof(int) * (size_t)nt, st));
        if (n > 0) {
            if (!device) CK(cudaMemcpyAsync(c->in_xyz.p, xyz, sizeof(double) * 3 * (size_t)n, cudaMemcpyHostToDevice, st));
            k_cg_count<<<blocks, 256, 0, st>>>(G, dxyz, n, (int)gx, tcnt);
        }
        k_cg_offsets<<<1, 1024, 0, st>>>(tcnt, nt, toff);
        if (n > 0) k_cg_fill<<<blocks, 256, 0, st>>>(G, dxyz, n, (int)gx, toff, tcnt, R);
        k_cg_sites<<<nt, 256, 0, st>>>(G, dxyz, (int)gx, (int)((span + kCgTile - 1) / kCgTile), toff, R, pixel);
    } else {
        const int ntx = (int)((xp + kCpTile - 1) / kCpTile), nty = (int)((yp + kCpTile - 1) / kCpTile);
        const int nt = ntx * nty;
        // tiles one square can reach
        const long long per = (span / kCpTile + 2) * (span / kCpTile + 2);
        const int64_t list_n = std::max<int64_t>(n * per, 1);
        if ((rs = dnni_ensure(c, c->scr.cnt, tile_bytes(nt, 2))) ||
            (rs = dnni_ensure(c, c->scr.list, sizeof(uint32_t) * (size_t)list_n)))
            return rs;
        long long* toff = (long long*)c->scr.cnt.p;
        int* tcnt = (int*)(toff + nt + 1);
        int* tcur = tcnt + nt;
        CK(cudaMemsetAsync(tcnt, 0, sizeof(int) * (size_t)nt, st));
        if (n > 0) {
            if (!device) CK(cudaMemcpyAsync(c->in_xyz.p, xyz, sizeof(double) * 3 * (size_t)n, cudaMemcpyHostToDevice, st));
            k_compat_count<<<c->sm_count * 8, 256, 0, st>>>(G, dxyz, n, ntx, tcnt);
        }
        k_compat_offsets<<<1, 1024, 0, st>>>(tcnt, nt, toff, tcur);
        if (n > 0)
            k_compat_fill<<<c->sm_count * 8, 256, 0, st>>>(G, dxyz, n, ntx, toff, tcur, (uint32_t*)c->scr.list.p, list_n);
        CK(cudaFuncSetAttribute(k_compat_sites, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kCpTileSmem));
        k_compat_sites<<<nt, 256, kCpTileSmem, st>>>(G, dxyz, ntx, toff, (const uint32_t*)c->scr.list.p, list_n, pixel);
    }
    k_compat_cells<<<(int)((cells + 255) / 256), 256, 0, st>>>(G, pixel, dh, dres);
    CK(cudaGetLastError());
    if (!device) {
        CK(cudaMemcpyAsync(h_out, c->out_h.p, sizeof(float) * (size_t)cells, cudaMemcpyDeviceToHost, st));
        if (res_out)
            CK(cudaMemcpyAsync(res_out, c->out_site.p, sizeof(int32_t) * (size_t)cells, cudaMemcpyDeviceToHost, st));
        CK(cudaStreamSynchronize(st));
    }
    return DNNI_OK;
}

extern "C" dnni_status dnni_interpolate_compat(dnni_ctx* c, const dnni_compat_settings* s, const dnni_compat_wp* wp,
                                               const double* xyz, int64_t n, float* h_out, int32_t* res_out) {
    if (!c || !s || !wp || !h_out || n < 0 || (n > 0 && !xyz)) return DNNI_E_INVAL;
    c->err.clear();
    DeviceGuard g(c->device);
    return with_room(c, [&] { return compat_run(c, s, wp, xyz, n, h_out, res_out, false, c->stream); });
}

extern "C" dnni_status dnni_interpolate_compat_device(dnni_ctx* c, const dnni_compat_settings* s,
                                                      const dnni_compat_wp* wp, const double* d_xyz, int64_t n,
                                                      float* d_h, int32_t* d_res, void* stream) {
    if (!c || !s || !wp || !d_h || n < 0 || (n > 0 && !d_xyz)) return DNNI_E_INVAL;
    c->err.clear();
    DeviceGuard g(c->device);
    const cudaStream_t st = stream ? (cudaStream_t)stream : c->stream;
    return with_room(c, [&] { return compat_run(c, s, wp, d_xyz, n, d_h, d_res, true, st); });
}
