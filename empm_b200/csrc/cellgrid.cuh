// cellgrid.cuh — point sets sorted into uniform cell grids, and exact nearest
// neighbour search in them.
//
// A brute-force search looks at every point for every query: 25 G distances for
// 500k queries among 50k points, 18.2 ms at the issue limit. Here the points of
// each set are counting-sorted into a grid of cubic cells over their bounding box
// (a few points per cell, at most 1024 cells per axis), and a query visits the
// cells around its own until it has k neighbours, then those that the ball through the
// k-th of them reaches. Queries run in cell order as well, so that the lanes of a warp
// visit the same cells together.
//
// 500k queries among 50k points, k = 16: 0.65 ms for the search (0.77 with the k best
// in local memory) and 0.05 ms for the sorting, bound by the insertions of candidates,
// which one lane or another of a warp makes for nearly every point it looks at.
//
// 80,000 queries and points, both searches of a chamfer distance (brute force 6.5 ms)
// and k = 16 (6.3 ms), with cells left out ring by ring by one axis at a time before:
//   the same cube             0.09 ms (0.09)    0.22 ms (0.29)
//   cubes side by side        0.11 (38)         0.33 (21)
//   over a sheet of 20,000    0.10 (21)         0.18 (8)
//   one point far away        6.6 (9.7)         4.5 (25)
//   most points in one cell   6.9 (23)          4.5 (42)
//
// Results are those of the brute-force search bit for bit: the same distance
// expression, ties in index order, and points or queries that are not finite have
// no neighbours. Several sets (the clouds of many chamfer pairs) are handled by
// the same launches.
#pragma once
#include <cuda_runtime.h>
#include <float.h>
#include <math.h>

namespace empm {

// Squared distance, spelled out so that every search forms it alike: the order in
// which the compiler contracts dx * dx + dy * dy + dz * dz, which decides between
// neighbours whose distances differ in the last bit.
__device__ __forceinline__ float point_dist2(float qx, float qy, float qz, float px, float py, float pz) {
    const float dx = qx - px, dy = qy - py, dz = qz - pz;
    return __fmaf_rn(dz, dz, __fmaf_rn(dx, dx, __fmul_rn(dy, dy)));
}

struct SetGrid {
    float lo[3], ext[3];   // corner and extent of the box
    float h, inv_h;
    int   dim[3];
    int   cells;
    int   base;      // first of the set's cells + 1 bins (the last bin: points that are not finite)
    int   first;     // first of the set's points in the sorted array
};

// Up to two arrays of sets: set s < n_a is rows [a_off[s], a_off[s + 1]) of a, the
// others those of b. Offsets NULL: one set of all rows.
struct PointSets {
    const float* a; const int* a_off; int sets_a, rows_a;
    const float* b; const int* b_off; int sets_b, rows_b;
    __host__ __device__ int sets() const { return sets_a + sets_b; }
    __host__ __device__ int rows() const { return rows_a + rows_b; }
};

__device__ __forceinline__ int set_find(const int* off, int n, int i) {
    if (!off) return 0;
    int lo = 0, hi = n - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (__ldg(off + mid) <= i) lo = mid; else hi = mid - 1;
    }
    return lo;
}

// set, coordinates and row (within a or b) of point i of all sets
__device__ __forceinline__ int set_point(const PointSets& P, int i, float& x, float& y, float& z, int& row) {
    const bool in_a = i < P.rows_a;
    row = in_a ? i : i - P.rows_a;
    const float* src = (in_a ? P.a : P.b) + 3 * (size_t)row;
    x = __ldg(src);
    y = __ldg(src + 1);
    z = __ldg(src + 2);
    return in_a ? set_find(P.a_off, P.sets_a, row) : P.sets_a + set_find(P.b_off, P.sets_b, row);
}

// order-preserving code of a float as unsigned
__device__ __forceinline__ unsigned float_code(float f) {
    const unsigned u = __float_as_uint(f);
    return u & 0x80000000u ? ~u : u | 0x80000000u;
}
__device__ __forceinline__ float float_decode(unsigned u) {
    return __uint_as_float(u & 0x80000000u ? u & 0x7fffffffu : ~u);
}

static __global__ void k_box_init(unsigned* box, int n6) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n6) box[i] = (i % 6) < 3 ? 0xffffffffu : 0u;
}

// Bounding boxes of the finite points, 512 points per warp: one set of atomics
// per warp and set (two of a million points, 2 k of them, meet on a word).
static __global__ void __launch_bounds__(256) k_box(const PointSets P, int n, unsigned* box) {
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    unsigned v[6] = {0xffffffffu, 0xffffffffu, 0xffffffffu, 0u, 0u, 0u};
    int cur = -1;   // the set the accumulated box belongs to (the same in every lane)
    auto flush = [&]() {
        if (cur < 0) return;
#pragma unroll
        for (int e = 0; e < 6; ++e) {
            const unsigned r = e < 3 ? __reduce_min_sync(0xffffffffu, v[e]) : __reduce_max_sync(0xffffffffu, v[e]);
            if (lane == 0) { if (e < 3) atomicMin(box + 6 * cur + e, r); else atomicMax(box + 6 * cur + e, r); }
            v[e] = e < 3 ? 0xffffffffu : 0u;
        }
    };
    for (int it = 0; it < 16; ++it) {
        const int i = (warp * 16 + it) * 32 + lane;
        float x = 0.f, y = 0.f, z = 0.f;
        int s = -1, row;
        if (i < n) s = set_point(P, i, x, y, z, row);
        const bool ok = i < n && isfinite(x) && isfinite(y) && isfinite(z);
        const unsigned c[3] = {float_code(x), float_code(y), float_code(z)};
        const int s0 = __shfl_sync(0xffffffffu, s, 0);
        if (__all_sync(0xffffffffu, s == s0 || s < 0)) {
            if (s0 != cur) { flush(); cur = s0; }
            if (ok)
#pragma unroll
                for (int e = 0; e < 3; ++e) { v[e] = min(v[e], c[e]); v[3 + e] = max(v[3 + e], c[e]); }
        } else if (ok) {   // the boundary of two sets
#pragma unroll
            for (int e = 0; e < 3; ++e) { atomicMin(box + 6 * s + e, c[e]); atomicMax(box + 6 * s + 3 + e, c[e]); }
        }
    }
    flush();
}

// Grid of each set: cubic cells with about `per_cell` points, axes thinner than a
// cell left whole. share: set 1 uses set 0's grid (queries binned like the points).
static __global__ void k_grid_setup(const PointSets P, const unsigned* box, SetGrid* grids, float per_cell, int share) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= P.sets()) return;
    const bool in_a = s < P.sets_a;
    const int* off = in_a ? P.a_off : P.b_off;
    const int ls = in_a ? s : s - P.sets_a;
    const int first = off ? off[ls] : 0;
    const int n = off ? off[ls + 1] - first : (in_a ? P.rows_a : P.rows_b);
    const int src = share ? 0 : s;
    const int n_src = share ? P.rows_a : n;
    SetGrid g;
    const int at = in_a ? first : P.rows_a + first;
    g.first = at;
    g.base = share ? s * (P.rows_a / 2 + 2) : at / 2 + 2 * s;
    float ext[3];
    bool ok = true;
    for (int a = 0; a < 3; ++a) {
        const unsigned lo = box[6 * src + a], hi = box[6 * src + 3 + a];
        ok = ok && lo <= hi;
        g.lo[a] = ok ? float_decode(lo) : 0.f;
        ext[a] = ok ? float_decode(hi) - g.lo[a] : 0.f;
        ok = ok && ext[a] < 1e30f;
        g.dim[a] = 1;
    }
    for (int a = 0; a < 3; ++a) g.ext[a] = ext[a];
    g.cells = 1;
    g.h = 1.f;
    const float want = fmaxf(1.f, fminf((float)n_src / per_cell, (float)(n_src / 2)));
    const float longest = fmaxf(ext[0], fmaxf(ext[1], ext[2]));
    if (ok && longest > 1e-30f && want >= 2.f) {
        // h from the volume over the axes longer than h
        float h = longest;
        for (int axes = 3; axes >= 1; --axes) {
            float log_sum = 0.f;
            int used = 0;
            for (int a = 0; a < 3; ++a)
                if (ext[a] > h * 1e-6f && (axes == 3 || ext[a] >= h)) { log_sum += logf(ext[a]); ++used; }
            h = used ? expf((log_sum - logf(want)) / used) : longest;
            if (ext[0] >= h && ext[1] >= h && ext[2] >= h) break;
        }
        h = fmaxf(h, longest / 1020.f);
        for (int it = 0; it < 200; ++it) {
            float total = 1.f;
            for (int a = 0; a < 3; ++a) total *= floorf(ext[a] / h) + 1.f;
            if (total <= (float)(n_src / 2)) break;
            h *= 1.02f;
        }
        int total = 1;
        const float inv = 1.f / h;
        int d[3];
        for (int a = 0; a < 3; ++a) { d[a] = min(1023, (int)(ext[a] * inv)) + 1; }
        const long long cells = (long long)d[0] * d[1] * d[2];
        if (cells <= n_src / 2) {
            for (int a = 0; a < 3; ++a) g.dim[a] = d[a];
            total = (int)cells;
            g.h = h;
        }
        g.cells = total;
    }
    g.inv_h = 1.f / g.h;
    grids[s] = g;
}

__device__ __forceinline__ int cell_axis(float x, float lo, float inv_h, int dim) {
    return min(max((int)floorf((x - lo) * inv_h), 0), dim - 1);
}

__device__ __forceinline__ int cell_bin(const SetGrid& g, float x, float y, float z) {
    if (!(isfinite(x) && isfinite(y) && isfinite(z))) return g.base + g.cells;
    if (g.cells == 1) return g.base;
    return g.base + (cell_axis(x, g.lo[0], g.inv_h, g.dim[0]) * g.dim[1] + cell_axis(y, g.lo[1], g.inv_h, g.dim[1])) *
                        g.dim[2] + cell_axis(z, g.lo[2], g.inv_h, g.dim[2]);
}

// start[c + 1] counts bin c
static __global__ void __launch_bounds__(256) k_bin_count(const PointSets P, int n, const SetGrid* grids, int* start) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float x, y, z;
    int row;
    const int s = set_point(P, i, x, y, z, row);
    atomicAdd(start + 1 + cell_bin(grids[s], x, y, z), 1);
}

constexpr int kScanTile = 2048;

static __global__ void __launch_bounds__(256) k_scan_sums(const int* v, int n, int* sums) {
    __shared__ int part[8];
    const int t = threadIdx.x;
    int s = 0;
#pragma unroll
    for (int e = 0; e < 8; ++e) {
        const int i = blockIdx.x * kScanTile + e * 256 + t;
        if (i < n) s += v[i];
    }
    s = __reduce_add_sync(0xffffffffu, s);
    if ((t & 31) == 0) part[t >> 5] = s;
    __syncthreads();
    if (t == 0) {
        int total = 0;
        for (int w = 0; w < 8; ++w) total += part[w];
        sums[blockIdx.x] = total;
    }
}

// exclusive scan of one value per thread over a block of 256; total gets the sum
__device__ __forceinline__ int block_scan(int v, int* part, int& total) {
    const int t = threadIdx.x, lane = t & 31;
    int incl = v;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const int up = __shfl_up_sync(0xffffffffu, incl, d);
        if (lane >= d) incl += up;
    }
    __syncthreads();
    if (lane == 31) part[t >> 5] = incl;
    __syncthreads();
    int before = 0;
    total = 0;
#pragma unroll
    for (int w = 0; w < 8; ++w) {
        if (w < (t >> 5)) before += part[w];
        total += part[w];
    }
    return before + incl - v;
}

static __global__ void __launch_bounds__(256) k_scan_top(int* sums, int n) {
    __shared__ int part[8];
    int carry = 0;
    for (int b = 0; b < n; b += 256) {
        const int i = b + threadIdx.x;
        int total;
        const int ex = block_scan(i < n ? sums[i] : 0, part, total);
        if (i < n) sums[i] = carry + ex;
        carry += total;
    }
}

// v[i] <- exclusive sum
static __global__ void __launch_bounds__(256) k_scan_apply(int* v, int n, const int* sums) {
    __shared__ int part[8];
    const int i0 = blockIdx.x * kScanTile + threadIdx.x * 8;
    int e[8], s = 0;
#pragma unroll
    for (int k = 0; k < 8; ++k) { e[k] = i0 + k < n ? v[i0 + k] : 0; s += e[k]; }
    int total;
    int at = sums[blockIdx.x] + block_scan(s, part, total);
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        if (i0 + k < n) v[i0 + k] = at;
        at += e[k];
    }
}

// Points to their bins: (x, y, z, row). Afterwards bin c holds
// sorted[start[c] .. start[c + 1]) (start[0] is 0).
static __global__ void __launch_bounds__(256) k_bin_scatter(const PointSets P, int n, const SetGrid* grids, int* start,
                                                     float4* sorted) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float x, y, z;
    int row;
    const int s = set_point(P, i, x, y, z, row);
    const int at = atomicAdd(start + 1 + cell_bin(grids[s], x, y, z), 1);
    sorted[at] = make_float4(x, y, z, __int_as_float(row));
}

// ---- workspace ----------------------------------------------------------------
struct CellGridWork {
    SetGrid*  grids;
    unsigned* box;
    double*   acc;      // one per set, zero after the build
    int*      start;    // bins + 1
    int*      sums;
    float4*   sorted;
    int*      rest;     // per set: queries that the cells are no use to
    int*      rest_row; // their rows, from the set's first on
    int       bins;
    float     per_cell;
};

// The parts of a workspace for sets of `rows` points in all (share: query set
// binned in the point set's grid); base NULL: only the size.
inline size_t cellgrid_layout(const PointSets& P, int share, float per_cell, void* base, CellGridWork* w) {
    const long long bins = share ? 2LL * (P.rows_a / 2 + 2) : (long long)P.rows() / 2 + 2LL * P.sets() + 2;
    size_t at = 0;
    auto take = [&](size_t bytes) {
        const size_t here = at;
        at += (bytes + 255) & ~(size_t)255;
        return base ? (char*)base + here : nullptr;
    };
    CellGridWork c;
    c.grids = (SetGrid*)take(sizeof(SetGrid) * P.sets());
    c.box = (unsigned*)take(sizeof(unsigned) * 6 * P.sets());
    c.acc = (double*)take(sizeof(double) * P.sets() + sizeof(int) * (bins + 1 + P.sets()));
    c.start = base ? (int*)(c.acc + P.sets()) : nullptr;
    c.rest = base ? c.start + bins + 1 : nullptr;
    c.rest_row = (int*)take(sizeof(int) * (size_t)P.rows());
    c.sums = (int*)take(sizeof(int) * (bins / kScanTile + 1));
    c.sorted = (float4*)take(sizeof(float4) * (size_t)P.rows());
    c.bins = (int)bins;
    c.per_cell = per_cell;
    if (w) *w = c;
    return at;
}

// Sorts the sets into w (all launches on s).
inline cudaError_t cellgrid_build(const PointSets& P, int share, const CellGridWork& w,
                                  cudaStream_t s) {
    const int n = P.rows(), sets = P.sets();
    const auto blocks = [](long long k, int t) { return (unsigned)((k + t - 1) / t); };
    cudaError_t e = cudaMemsetAsync(w.acc, 0, sizeof(double) * sets + sizeof(int) * ((size_t)w.bins + 1 + sets), s);
    if (e != cudaSuccess) return e;
    k_box_init<<<blocks(6LL * sets, 256), 256, 0, s>>>(w.box, 6 * sets);
    k_box<<<blocks(n, 256 * 16), 256, 0, s>>>(P, n, w.box);
    k_grid_setup<<<blocks(sets, 64), 64, 0, s>>>(P, w.box, w.grids, w.per_cell, share);
    k_bin_count<<<blocks(n, 256), 256, 0, s>>>(P, n, w.grids, w.start);
    const int tiles = (int)blocks(w.bins, kScanTile);
    k_scan_sums<<<tiles, 256, 0, s>>>(w.start + 1, w.bins, w.sums);
    k_scan_top<<<1, 256, 0, s>>>(w.sums, tiles);
    k_scan_apply<<<tiles, 256, 0, s>>>(w.start + 1, w.bins, w.sums);
    k_bin_scatter<<<blocks(n, 256), 256, 0, s>>>(P, n, w.grids, w.start, w.sorted);
    return cudaGetLastError();
}

// ---- search -------------------------------------------------------------------
// The KT nearest so far, in order of (distance, index).
template <int KT>
struct Nearest {
    float d[KT];
    int   i[KT];
    __device__ __forceinline__ void clear(float none) {
#pragma unroll
        for (int s = 0; s < KT; ++s) { d[s] = none; i[s] = -1; }
    }
    // a candidate with dist <= d[KT - 1]
    __device__ __forceinline__ void insert(float dist, int idx) {
        bool before = dist < d[KT - 1] || (dist == d[KT - 1] && idx < i[KT - 1]);
        if (!before) return;
#pragma unroll
        for (int s = KT - 1; s > 0; --s) {
            const bool up = dist < d[s - 1] || (dist == d[s - 1] && idx < i[s - 1]);
            d[s] = up ? d[s - 1] : (before ? dist : d[s]);
            i[s] = up ? i[s - 1] : (before ? idx : i[s]);
            before = up;
        }
        if (before) { d[0] = dist; i[0] = idx; }
    }
    __device__ __forceinline__ float kth(int k) const {
        float r = d[KT - 1];
#pragma unroll
        for (int s = 0; s < KT - 1; ++s) {
            const float ds = d[s];   // read first: a choice between addresses would put d into local memory
            if (s == k - 1) r = ds;
        }
        return r;
    }
};

// Points sorted[j .. e) to best, four at a time so that their loads are not waited for one
// by one (lists of 32, whose insertions dwarf the loads, one at a time).
template <int KT>
__device__ __forceinline__ void nearest_scan(const float4* __restrict__ sorted, int j, int e, float qx, float qy,
                                             float qz, int skip, Nearest<KT>& best) {
    if (KT <= 16) {
        for (; j + 4 <= e; j += 4) {
            float d[4];
            int row[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const float4 p = __ldg(sorted + j + u);
                d[u] = point_dist2(qx, qy, qz, p.x, p.y, p.z);
                row[u] = __float_as_int(p.w);
            }
            if (fminf(fminf(d[0], d[1]), fminf(d[2], d[3])) <= best.d[KT - 1]) {
#pragma unroll
                for (int u = 0; u < 4; ++u)
                    if (d[u] <= best.d[KT - 1] && row[u] != skip) best.insert(d[u], row[u]);
            }
        }
    }
    for (; j < e; ++j) {
        const float4 p = __ldg(sorted + j);
        const float d = point_dist2(qx, qy, qz, p.x, p.y, p.z);
        if (d <= best.d[KT - 1]) {
            const int row = __float_as_int(p.w);
            if (row != skip) best.insert(d, row);
        }
    }
}

// Distance on one axis from r (both from the box's corner) to the points of cell c: those
// of the last cell end at the box. Less the roundings of cell coordinates (1024
// cells 2^-23 each), generously.
__device__ __forceinline__ float cell_gap(float r, int c, int dim, float h, float ext) {
    const float below = c * h - r, above = r - (c == dim - 1 ? ext : (c + 1) * h);
    return fmaxf(fmaxf(below, above) - 1e-3f * h, 0.f);
}

// Squared distances that may be those of points nearer than d, squared too: both
// carry a few 2^-24 of themselves, below the normal numbers a few of the smallest ones.
__device__ __forceinline__ float ball_of(float d) { return d * 1.00001f + FLT_MIN; }

// The k nearest of a set's points to q, added to best (which starts clear with a
// distance that no candidate reaches). skip: row left out (-1: none).
// The cubes of 3, 7, 15 ... cells around q's until they hold k points; then, once, the
// cells that the ball through the k-th of them reaches. Cells are looked at as runs
// along z, which are contiguous, and left out by their distance to q on all three
// axes, so a query beside the points' box visits the part of its side that the ball
// touches, and one among clusters no ring after ring of empty cells.
//
// Returns false, best being incomplete, where the cells are no use, because the set's n
// points are crowded in a few of them (one outlier at a hundred times the others'
// extent does it): when the first cube holds more than half of them, or the later cells
// more than a quarter. The caller then leaves the query to brute force, which needs
// 0.4 to 0.8 of the time per point (its points come from shared memory).
template <int KT>
__device__ __forceinline__ bool nearest_search(const SetGrid& g, const int* __restrict__ start,
                                               const float4* __restrict__ sorted, float qx, float qy, float qz, int k,
                                               int skip, int n, Nearest<KT>& best) {
    if (!(isfinite(qx) && isfinite(qy) && isfinite(qz))) return true;
    const int dx = g.dim[0], dy = g.dim[1], dz = g.dim[2];
    const int cx = cell_axis(qx, g.lo[0], g.inv_h, dx), cy = cell_axis(qy, g.lo[1], g.inv_h, dy),
              cz = cell_axis(qz, g.lo[2], g.inv_h, dz);
    const float rx = qx - g.lo[0], ry = qy - g.lo[1], rz = qz - g.lo[2];
    const float slack = 1e-3f * g.h;
    const float out_z = fmaxf(fmaxf(-rz, rz - g.ext[2]) - slack, 0.f);
    int done = -1, r = 1;       // the cube of radius done has been visited, that of radius r is next
    bool ball = false;          // the pass over the ball's cells
    float reach = INFINITY;     // its squared radius
    int x0 = max(cx - r, 0), x1 = min(cx + r, dx - 1), y0 = max(cy - r, 0), y1 = min(cy + r, dy - 1),
        z0 = max(cz - r, 0), z1 = min(cz + r, dz - 1);
    // counted before any is looked at: most of a crowded set's queries are in its crowds
    int near = 0;
    for (int x = x0; x <= x1; ++x)
        for (int y = y0; y <= y1; ++y) {
            const int c = g.base + (x * dy + y) * dz;
            near += __ldg(start + c + z1 + 1) - __ldg(start + c + z0);
        }
    if (near > n / 2) return false;
    int left = n / 4;
    for (;;) {
        for (int x = x0; x <= x1; ++x) {
            float gx = 0.f;
            if (ball) {
                gx = cell_gap(rx, x, dx, g.h, g.ext[0]);
                reach = fminf(reach, ball_of(best.kth(k)));
                if (!(gx * gx + out_z * out_z <= reach)) continue;
            }
            for (int y = y0; y <= y1; ++y) {
                const bool inner = abs(x - cx) <= done && abs(y - cy) <= done;
                if (inner && z0 >= cz - done && z1 <= cz + done) {   // nothing new up to the cube's far side
                    y = min(cy + done, y1);
                    continue;
                }
                int za = z0, zb = z1;
                if (ball) {
                    const float gy = cell_gap(ry, y, dy, g.h, g.ext[1]);
                    const float d = gx * gx + gy * gy;
                    if (!(d + out_z * out_z <= reach)) continue;
                    if (reach <= FLT_MAX) {
                        const float w = sqrtf(reach - d) + slack;
                        za = max(za, (int)floorf((rz - w) * g.inv_h));
                        zb = min(zb, (int)floorf((rz + w) * g.inv_h));
                    }
                }
                const int c = g.base + (x * dy + y) * dz;
                for (int part = inner ? 0 : 1; part < 2; ++part) {
                    const int a = part && inner ? max(za, cz + done + 1) : za;
                    const int b = part ? zb : min(zb, cz - done - 1);
                    if (a > b) continue;
                    const int j = __ldg(start + c + a), e = __ldg(start + c + b + 1);
                    if (done >= 0 && (left -= e - j) < 0) return false;
                    nearest_scan<KT>(sorted, j, e, qx, qy, qz, skip, best);
                }
            }
        }
        if (ball || (x0 == 0 && x1 == dx - 1 && y0 == 0 && y1 == dy - 1 && z0 == 0 && z1 == dz - 1)) return true;
        done = r;
        const float kth = best.kth(k);
        if (kth < FLT_MAX) {
            ball = true;
            reach = ball_of(kth);
            const float w = sqrtf(reach) + slack;
            x0 = max((int)floorf((rx - w) * g.inv_h), 0);
            x1 = min((int)floorf((rx + w) * g.inv_h), dx - 1);
            y0 = max((int)floorf((ry - w) * g.inv_h), 0);
            y1 = min((int)floorf((ry + w) * g.inv_h), dy - 1);
            z0 = max((int)floorf((rz - w) * g.inv_h), 0);
            z1 = min((int)floorf((rz + w) * g.inv_h), dz - 1);
            if (x0 >= cx - done && x1 <= cx + done && y0 >= cy - done && y1 <= cy + done && z0 >= cz - done &&
                z1 <= cz + done)
                return true;
        } else {
            r = 2 * r + 1;
            x0 = max(cx - r, 0), x1 = min(cx + r, dx - 1), y0 = max(cy - r, 0), y1 = min(cy + r, dy - 1);
            z0 = max(cz - r, 0), z1 = min(cz + r, dz - 1);
        }
    }
}

}  // namespace empm
