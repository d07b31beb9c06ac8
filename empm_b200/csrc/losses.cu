// losses.cu — training losses on the device: batched chamfer distance and
// its gradient.
//
// The reference trainer scores a rollout with pytorch3d's chamfer_distance
// (phys_sim/engine/trainer_warp_mpm.py:542-561, 617-642, 745-765): for point
// sets X and Y, mean over x of min_y |x - y|^2 plus mean over y of
// min_x |x - y|^2 (point_reduction "mean"). Here many (X, Y) pairs (one per
// population member and frame) are scored in one launch: pair p owns
// X rows [x_off[p], x_off[p+1]) and Y rows [y_off[p], y_off[p+1]). The nearest
// neighbours are found exactly, in cell grids of the clouds (cellgrid.cuh) or, for
// small ones, by brute force over shared-memory tiles of the other set, with the
// same results, and kept for the gradient.
#include <cuda_runtime.h>
#include <float.h>
#include <stdint.h>
#include "../../include/empm_b200.h"
#include "cellgrid.cuh"
#include "ctx.hpp"

using namespace empm;

namespace {

constexpr int kThreads = 256;

inline int blocks_for(long long n, int threads) { return (int)((n + threads - 1) / threads); }

// For every query point q of pair blockIdx.y: nearest point of the pair's
// target set, its squared distance added to sum[pair]. rest: only the pair's first
// rest[pair] of the queries rest_row.
template <typename Sum>
__global__ void __launch_bounds__(kThreads) k_nn(const float* __restrict__ q, const int* __restrict__ q_off,
                                                 const float* __restrict__ t, const int* __restrict__ t_off,
                                                 int* __restrict__ nn, Sum* __restrict__ sum,
                                                 const int* __restrict__ rest, const int* __restrict__ rest_row) {
    __shared__ float4 tile[kThreads];
    const int pair = blockIdx.y;
    const int q0 = __ldg(q_off + pair), q1 = rest ? q0 + __ldg(rest + pair) : __ldg(q_off + pair + 1);
    const int t0 = __ldg(t_off + pair), t1 = __ldg(t_off + pair + 1);
    const int slot = q0 + blockIdx.x * kThreads + threadIdx.x;
    if (q0 + (int)(blockIdx.x * kThreads) >= q1) return;   // whole CTA beyond this pair's queries
    const bool live = slot < q1;
    const int i = live && rest ? __ldg(rest_row + slot) : slot;
    float qx = 0.f, qy = 0.f, qz = 0.f;
    if (live) { qx = __ldg(q + 3 * i); qy = __ldg(q + 3 * i + 1); qz = __ldg(q + 3 * i + 2); }
    float best = FLT_MAX;
    int arg = -1;
    for (int base = t0; base < t1; base += kThreads) {
        const int j = base + threadIdx.x;
        __syncthreads();
        tile[threadIdx.x] = j < t1 ? make_float4(__ldg(t + 3 * j), __ldg(t + 3 * j + 1), __ldg(t + 3 * j + 2), 0.f)
                                   : make_float4(FLT_MAX, FLT_MAX, FLT_MAX, 0.f);
        __syncthreads();
        const int m = min(kThreads, t1 - base);
        for (int k = 0; k < m; ++k) {
            const float4 p = tile[k];
            const float d = point_dist2(qx, qy, qz, p.x, p.y, p.z);
            if (d < best) { best = d; arg = base + k; }
        }
    }
    if (live) nn[i] = arg;
    // warp-level partial sums (every lane of the CTA is still here; lanes
    // without a query add zero), one atomic per warp
    Sum v = (live && arg >= 0) ? best : 0.f;
    for (int d = 16; d > 0; d >>= 1) v += __shfl_down_sync(0xffffffffu, v, d);
    if ((threadIdx.x & 31) == 0 && v != 0) atomicAdd(sum + pair, v);
}

// The same through cell grids: one thread per point of either cloud, in the order
// of its own cloud's cells, searching the other cloud of its pair. Clouds of the
// same size apart, the 27 cells around a query hold about 54 candidates. The sums are
// kept in 64 bits: in 32 their error was that of the order of the atomics, 1e-7 to
// 5e-7 from run to run for 100,000 points.
__global__ void __launch_bounds__(kThreads) k_nn_cells(const PointSets P, const CellGridWork w,
                                                       int* __restrict__ nn_x, int* __restrict__ nn_y) {
    __shared__ double part[kThreads / 32];
    __shared__ int ends[2];
    const int t = blockIdx.x * kThreads + threadIdx.x;
    const int n = P.rows();
    double v = 0.;
    int set = -1;
    if (t < n) {
        const bool in_a = t < P.rows_a;
        const int pair = in_a ? set_find(P.a_off, P.sets_a, t) : set_find(P.b_off, P.sets_b, t - P.rows_a);
        set = in_a ? pair : P.sets_a + pair;
        const float4 q = __ldg(w.sorted + t);
        Nearest<1> best;
        best.clear(FLT_MAX);
        const int* off = in_a ? P.b_off : P.a_off;
        if (nearest_search<1>(w.grids[in_a ? P.sets_a + pair : pair], w.start, w.sorted, q.x, q.y, q.z, 1, -1,
                              __ldg(off + pair + 1) - __ldg(off + pair), best)) {
            (in_a ? nn_x : nn_y)[__float_as_int(q.w)] = best.i[0];
            if (best.i[0] >= 0) v = best.d[0];
        } else {
            const int first = in_a ? __ldg(P.a_off + pair) : P.rows_a + __ldg(P.b_off + pair);
            w.rest_row[first + atomicAdd(w.rest + set, 1)] = __float_as_int(q.w);
        }
    }
    // one atomic per block; where clouds meet in it per warp, or per thread
    if (threadIdx.x == 0) ends[0] = set;
    if (threadIdx.x == min(kThreads, n - (int)(blockIdx.x * kThreads)) - 1) ends[1] = set;
    __syncthreads();
    const bool one = ends[0] == ends[1];
    if (!one && !__all_sync(0xffffffffu, set == __shfl_sync(0xffffffffu, set, 0) || set < 0)) {
        if (v != 0.) atomicAdd(w.acc + set, v);
        return;
    }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) v += __shfl_down_sync(0xffffffffu, v, d);
    if (!one) {
        if ((threadIdx.x & 31) == 0 && v != 0.) atomicAdd(w.acc + set, v);
        return;
    }
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = v;
    __syncthreads();
    if (threadIdx.x == 0) {
        double s = 0.;
        for (int k = 0; k < kThreads / 32; ++k) s += part[k];
        if (s != 0.) atomicAdd(w.acc + set, s);
    }
}

__global__ void k_sums(const double* __restrict__ acc, int n_pairs, float* __restrict__ sum_xy,
                       float* __restrict__ sum_yx) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= n_pairs) return;
    sum_xy[p] = (float)acc[p];
    sum_yx[p] = (float)acc[n_pairs + p];
}

// Gradient in X of  g_xy[p] * sum_i |x_i - y_nn(i)|^2 + g_yx[p] * sum_j |y_j - x_nn(j)|^2
__global__ void k_chamfer_grad_x(const float* __restrict__ x, const int* __restrict__ pair_of_x,
                                 const float* __restrict__ y, const int* __restrict__ nn_x,
                                 const float* __restrict__ g_xy, float* __restrict__ gx, int nx) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nx) return;
    const int j = nn_x[i];
    if (j < 0) return;
    const float g = 2.f * __ldg(g_xy + __ldg(pair_of_x + i));
    gx[3 * i] += g * (x[3 * i] - y[3 * j]);
    gx[3 * i + 1] += g * (x[3 * i + 1] - y[3 * j + 1]);
    gx[3 * i + 2] += g * (x[3 * i + 2] - y[3 * j + 2]);
}

__global__ void k_chamfer_grad_y_to_x(const float* __restrict__ x, const float* __restrict__ y,
                                      const int* __restrict__ pair_of_y, const int* __restrict__ nn_y,
                                      const float* __restrict__ g_yx, float* __restrict__ gx, int ny) {
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= ny) return;
    const int i = nn_y[j];
    if (i < 0) return;
    const float g = 2.f * __ldg(g_yx + __ldg(pair_of_y + j));
    atomicAdd(gx + 3 * i, g * (x[3 * i] - y[3 * j]));
    atomicAdd(gx + 3 * i + 1, g * (x[3 * i + 1] - y[3 * j + 1]));
    atomicAdd(gx + 3 * i + 2, g * (x[3 * i + 2] - y[3 * j + 2]));
}

__global__ void k_pair_index(const int* off, int n_pairs, int* pair_of, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    int lo = 0, hi = n_pairs - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (__ldg(off + mid) <= i) lo = mid; else hi = mid - 1;
    }
    pair_of[i] = lo;
}

}  // namespace

#define CKL(expr, what)                                                          \
    do {                                                                         \
        int _rc = empm_check_cuda(nullptr, (expr), what);                        \
        if (_rc != EMPM_OK) return _rc;                                          \
    } while (0)

// The brute-force search both ways. rest: only the queries left over by the cells
// (counts of the x clouds, then of the y clouds).
template <typename Sum>
static int launch_nn(const float* x, const int* x_off, int max_nx, const float* y, const int* y_off, int max_ny,
                     int n_pairs, Sum* sum_xy, Sum* sum_yx, int* nn_x, int* nn_y, const int* rest,
                     const int* rest_x, const int* rest_y, cudaStream_t s) {
    if (max_nx > 0) {
        k_nn<<<dim3(blocks_for(max_nx, kThreads), n_pairs), kThreads, 0, s>>>(x, x_off, y, y_off, nn_x, sum_xy, rest,
                                                                             rest_x);
        CKL(cudaGetLastError(), "k_nn (x -> y)");
    }
    if (max_ny > 0) {
        k_nn<<<dim3(blocks_for(max_ny, kThreads), n_pairs), kThreads, 0, s>>>(y, y_off, x, x_off, nn_y, sum_yx,
                                                                             rest ? rest + n_pairs : nullptr, rest_y);
        CKL(cudaGetLastError(), "k_nn (y -> x)");
    }
    return EMPM_OK;
}

static int check_chamfer(const float* x, const int* x_off, int nx, int max_nx, const float* y, const int* y_off, int ny,
                         int max_ny, int n_pairs, const float* sum_xy, const float* sum_yx, const int* nn_x,
                         const int* nn_y) {
    if (n_pairs < 1 || n_pairs > 65535 || nx < 0 || ny < 0 || max_nx < 0 || max_ny < 0)
        return empm_set_error(nullptr, EMPM_ERR_INVALID, "bad chamfer sizes (%d pairs)", n_pairs);
    if (!x_off || !y_off || !sum_xy || !sum_yx || (nx && (!x || !nn_x)) || (ny && (!y || !nn_y)))
        return empm_set_error(nullptr, EMPM_ERR_INVALID, "chamfer pointer is NULL");
    return EMPM_OK;
}

extern "C" int empm_chamfer_workspace(int nx, int max_nx, int ny, int max_ny, int n_pairs, size_t* bytes) {
    if (n_pairs < 1 || nx < 0 || ny < 0 || max_nx < 0 || max_ny < 0 || !bytes)
        return empm_set_error(nullptr, EMPM_ERR_INVALID, "bad chamfer sizes (%d pairs)", n_pairs);
    // The brute-force search looks at 2.2e12 pairs of points a second; the grids'
    // ten launches and the sorting take about 60 us before the search, as long as
    // 7e7 pairs in each direction.
    *bytes = 0;
    if ((double)n_pairs * max_nx * max_ny < 7e7 || (long long)nx + ny > (1LL << 30)) return EMPM_OK;
    const PointSets P{nullptr, nullptr, n_pairs, nx, nullptr, nullptr, n_pairs, ny};
    *bytes = cellgrid_layout(P, 0, 2.f, nullptr, nullptr);
    return EMPM_OK;
}

extern "C" int empm_chamfer_cells(const float* x, const int* x_off, int nx, int max_nx, const float* y,
                                  const int* y_off, int ny, int max_ny, int n_pairs, float* sum_xy, float* sum_yx,
                                  int* nn_x, int* nn_y, void* workspace, size_t workspace_bytes, void* stream) {
    const int rc = check_chamfer(x, x_off, nx, max_nx, y, y_off, ny, max_ny, n_pairs, sum_xy, sum_yx, nn_x, nn_y);
    if (rc) return rc;
    size_t need = 0;
    empm_chamfer_workspace(nx, max_nx, ny, max_ny, n_pairs, &need);
    if (need == 0)
        return empm_chamfer(x, x_off, nx, max_nx, y, y_off, ny, max_ny, n_pairs, sum_xy, sum_yx, nn_x, nn_y, stream);
    if (!workspace || workspace_bytes < need || ((uintptr_t)workspace & 255))
        return empm_set_error(nullptr, EMPM_ERR_INVALID, "chamfer: workspace of %zu bytes, 256-byte aligned, needed",
                              need);
    cudaStream_t s = (cudaStream_t)stream;
    const PointSets P{x, x_off, n_pairs, nx, y, y_off, n_pairs, ny};
    CellGridWork w;
    cellgrid_layout(P, 0, 2.f, workspace, &w);
    CKL(cellgrid_build(P, 0, w, s), "chamfer cell grids");
    k_nn_cells<<<blocks_for((long long)nx + ny, kThreads), kThreads, 0, s>>>(P, w, nn_x, nn_y);
    CKL(cudaGetLastError(), "k_nn_cells");
    const int rn = launch_nn(x, x_off, max_nx, y, y_off, max_ny, n_pairs, w.acc, w.acc + n_pairs, nn_x, nn_y, w.rest,
                             w.rest_row, w.rest_row + nx, s);
    if (rn) return rn;
    k_sums<<<blocks_for(n_pairs, 256), 256, 0, s>>>(w.acc, n_pairs, sum_xy, sum_yx);
    CKL(cudaGetLastError(), "k_sums");
    return EMPM_OK;
}

extern "C" int empm_chamfer(const float* x, const int* x_off, int nx, int max_nx, const float* y, const int* y_off,
                            int ny, int max_ny, int n_pairs, float* sum_xy, float* sum_yx, int* nn_x, int* nn_y,
                            void* stream) {
    const int rc = check_chamfer(x, x_off, nx, max_nx, y, y_off, ny, max_ny, n_pairs, sum_xy, sum_yx, nn_x, nn_y);
    if (rc) return rc;
    cudaStream_t s = (cudaStream_t)stream;
    CKL(cudaMemsetAsync(sum_xy, 0, sizeof(float) * n_pairs, s), "chamfer");
    CKL(cudaMemsetAsync(sum_yx, 0, sizeof(float) * n_pairs, s), "chamfer");
    return launch_nn(x, x_off, max_nx, y, y_off, max_ny, n_pairs, sum_xy, sum_yx, nn_x, nn_y, nullptr, nullptr, nullptr, s);
}

extern "C" int empm_chamfer_backward(const float* x, const int* x_off, int nx, const float* y, const int* y_off,
                                     int ny, int n_pairs, const int* nn_x, const int* nn_y, const float* g_xy,
                                     const float* g_yx, float* grad_x, int* scratch_pair, void* stream) {
    if (n_pairs < 1 || nx < 0 || ny < 0)
        return empm_set_error(nullptr, EMPM_ERR_INVALID, "bad chamfer sizes (%d pairs)", n_pairs);
    if (!x_off || !y_off || !g_xy || !g_yx || !grad_x || !scratch_pair || (nx && (!x || !nn_x)) ||
        (ny && (!y || !nn_y)))
        return empm_set_error(nullptr, EMPM_ERR_INVALID, "chamfer pointer is NULL");
    cudaStream_t s = (cudaStream_t)stream;
    if (nx > 0) {
        k_pair_index<<<blocks_for(nx, 256), 256, 0, s>>>(x_off, n_pairs, scratch_pair, nx);
        CKL(cudaGetLastError(), "k_pair_index");
        k_chamfer_grad_x<<<blocks_for(nx, 256), 256, 0, s>>>(x, scratch_pair, y, nn_x, g_xy, grad_x, nx);
        CKL(cudaGetLastError(), "k_chamfer_grad_x");
    }
    if (ny > 0) {
        // the pair index of Y rows reuses the scratch after the X pass (stream order)
        k_pair_index<<<blocks_for(ny, 256), 256, 0, s>>>(y_off, n_pairs, scratch_pair, ny);
        CKL(cudaGetLastError(), "k_pair_index");
        k_chamfer_grad_y_to_x<<<blocks_for(ny, 256), 256, 0, s>>>(x, y, scratch_pair, nn_y, g_yx, grad_x, ny);
        CKL(cudaGetLastError(), "k_chamfer_grad_y_to_x");
    }
    return EMPM_OK;
}
