// knn.cu — exact k nearest neighbours (k <= 32).
//
// get_topk_indices and knn_weights_sparse of the reference
// (third_party/gaussian_splatting/dynamic_utils.py:248-265, 295-302) build dense
// distance matrices and call torch.topk. Small sets are searched by brute force
// through shared-memory tiles; larger ones in a cell grid (cellgrid.cuh), with the
// same results.
#include <cuda_runtime.h>
#include <math.h>
#include "../../include/empm_b200.h"
#include "cellgrid.cuh"
#include "ctx.hpp"

using namespace empm;

namespace {

inline int blocks_for(long long n, int threads) { return (int)((n + threads - 1) / threads); }
bool idx_ok(int idx_bytes) { return idx_bytes == 4 || idx_bytes == 8; }

// ---------------------------------------------------------------------------
// k nearest neighbours: one query per thread, candidates staged through
// shared memory, the KT best kept sorted in registers. rest: only the *rest
// queries rest_row.
// ---------------------------------------------------------------------------
constexpr int kKnnThreads = 128;
constexpr int kKnnTile = 1024;

template <int KT, typename IdxT>
__global__ void __launch_bounds__(kKnnThreads) k_knn(const float* __restrict__ q, int nq, const float* __restrict__ pts,
                                                     int np, int k, int exclude_self, IdxT* __restrict__ out_idx,
                                                     float* __restrict__ out_dist, const int* __restrict__ rest,
                                                     const int* __restrict__ rest_row) {
    __shared__ float4 tile[kKnnTile];
    if (rest) nq = *rest;
    if (blockIdx.x * kKnnThreads >= nq) return;
    const int t0 = blockIdx.x * kKnnThreads + threadIdx.x;
    const bool live = t0 < nq;
    const int i = live && rest ? __ldg(rest_row + t0) : t0;
    float qx = 0.f, qy = 0.f, qz = 0.f;
    if (live) { qx = __ldg(q + 3 * (long long)i); qy = __ldg(q + 3 * (long long)i + 1); qz = __ldg(q + 3 * (long long)i + 2); }
    float bd[KT];
    int bi[KT];
#pragma unroll
    for (int s = 0; s < KT; ++s) { bd[s] = INFINITY; bi[s] = -1; }
    const int self = (live && exclude_self) ? i : -1;
    for (int base = 0; base < np; base += kKnnTile) {
        const int m = min(kKnnTile, np - base);
        __syncthreads();
        for (int t = threadIdx.x; t < m; t += kKnnThreads) {
            const long long j = base + t;
            tile[t] = make_float4(__ldg(pts + 3 * j), __ldg(pts + 3 * j + 1), __ldg(pts + 3 * j + 2), 0.f);
        }
        __syncthreads();
        // insertion keeps equal distances in index order (strict <)
        const auto look = [&](float d, int j) {
            if (d < bd[KT - 1] && j != self) {
#pragma unroll
                for (int s = KT - 1; s > 0; --s) {
                    if (d < bd[s - 1]) { bd[s] = bd[s - 1]; bi[s] = bi[s - 1]; }
                    else if (d < bd[s]) { bd[s] = d; bi[s] = j; }
                }
                if (d < bd[0]) { bd[0] = d; bi[0] = j; }
            }
        };
        int t = 0;
        // four at a time: a thread's candidates are a chain of dependent waits else
        // (80,000 among 80,000, k = 16: 6.3 -> 4.1 ms; one query among 10,000 the same)
        if (KT <= 16) {
            for (; t + 4 <= m; t += 4) {
                float d[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const float4 p = tile[t + u];
                    d[u] = point_dist2(qx, qy, qz, p.x, p.y, p.z);
                }
                if (fminf(fminf(d[0], d[1]), fminf(d[2], d[3])) < bd[KT - 1]) {
#pragma unroll
                    for (int u = 0; u < 4; ++u) look(d[u], base + t + u);
                }
            }
        }
        for (; t < m; ++t) {
            const float4 p = tile[t];
            look(point_dist2(qx, qy, qz, p.x, p.y, p.z), base + t);
        }
    }
    if (!live) return;
#pragma unroll
    for (int s = 0; s < KT; ++s) {
        if (s < k) {
            out_idx[(long long)i * k + s] = (IdxT)bi[s];
            if (out_dist) out_dist[(long long)i * k + s] = sqrtf(bd[s]);
        }
    }
}

template <typename IdxT>
int launch_knn(const float* q, int nq, const float* pts, int np, int k, int exclude_self, IdxT* idx, float* dist,
               const int* rest, const int* rest_row, cudaStream_t s) {
    const int g = blocks_for(nq, kKnnThreads);
    if (k <= 8) k_knn<8, IdxT><<<g, kKnnThreads, 0, s>>>(q, nq, pts, np, k, exclude_self, idx, dist, rest, rest_row);
    else if (k <= 16) k_knn<16, IdxT><<<g, kKnnThreads, 0, s>>>(q, nq, pts, np, k, exclude_self, idx, dist, rest, rest_row);
    else k_knn<32, IdxT><<<g, kKnnThreads, 0, s>>>(q, nq, pts, np, k, exclude_self, idx, dist, rest, rest_row);
    return empm_check_cuda(nullptr, cudaGetLastError(), "k_knn");
}

// ---------------------------------------------------------------------------
// the same in a cell grid, one query per thread in cell order
// ---------------------------------------------------------------------------
template <int KT, typename IdxT>
__global__ void __launch_bounds__(kKnnThreads) k_knn_cells(const CellGridWork w, int first, int nq, int np, int k,
                                                           int exclude_self, IdxT* __restrict__ out_idx,
                                                           float* __restrict__ out_dist) {
    const int t = blockIdx.x * kKnnThreads + threadIdx.x;
    if (t >= nq) return;
    const float4 q = __ldg(w.sorted + first + t);
    const int row = __float_as_int(q.w);
    Nearest<KT> best;
    best.clear(INFINITY);
    if (!nearest_search<KT>(w.grids[0], w.start, w.sorted, q.x, q.y, q.z, k, exclude_self ? row : -1,
                            np, best)) {
        w.rest_row[atomicAdd(w.rest, 1)] = row;
        return;
    }
#pragma unroll
    for (int s = 0; s < KT; ++s) {
        if (s < k) {
            out_idx[(long long)row * k + s] = (IdxT)best.i[s];
            if (out_dist) out_dist[(long long)row * k + s] = sqrtf(best.d[s]);
        }
    }
}

template <typename IdxT>
int launch_knn_cells(const float* q, int nq, const float* pts, int np, int k, int exclude_self, IdxT* idx, float* dist,
                     void* workspace, cudaStream_t s) {
    const bool self = exclude_self != 0;   // the queries are the points
    const PointSets P{pts, nullptr, 1, np, self ? nullptr : q, nullptr, self ? 0 : 1, self ? 0 : nq};
    CellGridWork w;
    // about k / 3 points per cell: the 27 cells around a query then hold 9 k, and
    // mostly the k nearest among them
    cellgrid_layout(P, !self, fmaxf(2.f, k / 3.f), workspace, &w);
    cudaError_t e = cellgrid_build(P, !self, w, s);
    if (e != cudaSuccess) return empm_check_cuda(nullptr, e, "knn cell grid");
    const int first = self ? 0 : np, g = blocks_for(nq, kKnnThreads);
    if (k == 1) k_knn_cells<1, IdxT><<<g, kKnnThreads, 0, s>>>(w, first, nq, np, k, exclude_self, idx, dist);
    else if (k <= 8) k_knn_cells<8, IdxT><<<g, kKnnThreads, 0, s>>>(w, first, nq, np, k, exclude_self, idx, dist);
    else if (k <= 16) k_knn_cells<16, IdxT><<<g, kKnnThreads, 0, s>>>(w, first, nq, np, k, exclude_self, idx, dist);
    else k_knn_cells<32, IdxT><<<g, kKnnThreads, 0, s>>>(w, first, nq, np, k, exclude_self, idx, dist);
    const int rc = empm_check_cuda(nullptr, cudaGetLastError(), "k_knn_cells");
    return rc ? rc : launch_knn(q, nq, pts, np, k, exclude_self, idx, dist, w.rest, w.rest_row, s);
}

int check_knn(const float* queries, int n_queries, const float* points, int n_points, int k, int exclude_self,
              const void* out_idx, int idx_bytes) {
    if (n_queries < 0 || n_points < 0 || k < 1 || k > EMPM_KNN_MAX_K || !idx_ok(idx_bytes))
        return empm_set_error(nullptr, EMPM_ERR_INVALID, "knn: bad sizes (k %d, idx_bytes %d)", k, idx_bytes);
    if (exclude_self && n_queries != n_points)
        return empm_set_error(nullptr, EMPM_ERR_INVALID, "knn: exclude_self needs queries == points");
    if (k > n_points - (exclude_self ? 1 : 0))
        return empm_set_error(nullptr, EMPM_ERR_INVALID, "knn: k %d exceeds the %d candidates", k,
                              n_points - (exclude_self ? 1 : 0));
    if (n_queries > 0 && (!queries || !points || !out_idx))
        return empm_set_error(nullptr, EMPM_ERR_INVALID, "knn: NULL pointer");
    return EMPM_OK;
}

}  // namespace

extern "C" int empm_knn(const float* queries, int n_queries, const float* points, int n_points, int k,
                        int exclude_self, void* out_idx, int idx_bytes, float* out_dist, void* stream) {
    const int rc = check_knn(queries, n_queries, points, n_points, k, exclude_self, out_idx, idx_bytes);
    if (rc != EMPM_OK || n_queries == 0) return rc;
    cudaStream_t s = (cudaStream_t)stream;
    if (idx_bytes == 8)
        return launch_knn(queries, n_queries, points, n_points, k, exclude_self, (long long*)out_idx, out_dist,
                          nullptr, nullptr, s);
    return launch_knn(queries, n_queries, points, n_points, k, exclude_self, (int*)out_idx, out_dist, nullptr, nullptr,
                      s);
}

extern "C" int empm_knn_workspace(int n_queries, int n_points, int exclude_self, size_t* bytes) {
    if (n_queries < 0 || n_points < 0 || !bytes)
        return empm_set_error(nullptr, EMPM_ERR_INVALID, "knn workspace: bad arguments");
    // At 2,000 points, as many queries: brute force 127, 127, 173, 349 us for k = 1, 5,
    // 16, 32, the grid 59, 78, 112, 229 with its eleven launches; for one query, where a
    // thread's candidates are waited for one after another, 100 and 79 (k = 1), 139 and
    // 105 (k = 16). Below, brute force shrinks with the points (1,000: 65 us for k = 1)
    // and the launches stay.
    *bytes = 0;
    if (n_points < 2000 || n_queries < 1 || (long long)n_points + n_queries > (1LL << 30)) return EMPM_OK;
    const PointSets P{nullptr, nullptr, 1, n_points, nullptr, nullptr, exclude_self ? 0 : 1,
                      exclude_self ? 0 : n_queries};
    *bytes = cellgrid_layout(P, !exclude_self, 1.f, nullptr, nullptr);
    return EMPM_OK;
}

extern "C" int empm_knn_cells(const float* queries, int n_queries, const float* points, int n_points, int k,
                              int exclude_self, void* out_idx, int idx_bytes, float* out_dist, void* workspace,
                              size_t workspace_bytes, void* stream) {
    const int rc = check_knn(queries, n_queries, points, n_points, k, exclude_self, out_idx, idx_bytes);
    if (rc != EMPM_OK || n_queries == 0) return rc;
    size_t need = 0;
    empm_knn_workspace(n_queries, n_points, exclude_self, &need);
    // another query array than the points cannot share their bins
    if (need == 0 || (exclude_self && queries != points))
        return empm_knn(queries, n_queries, points, n_points, k, exclude_self, out_idx, idx_bytes, out_dist, stream);
    if (!workspace || workspace_bytes < need || ((uintptr_t)workspace & 255))
        return empm_set_error(nullptr, EMPM_ERR_INVALID, "knn: workspace of %zu bytes, 256-byte aligned, needed", need);
    cudaStream_t s = (cudaStream_t)stream;
    if (idx_bytes == 8)
        return launch_knn_cells(queries, n_queries, points, n_points, k, exclude_self, (long long*)out_idx, out_dist,
                                workspace, s);
    return launch_knn_cells(queries, n_queries, points, n_points, k, exclude_self, (int*)out_idx, out_dist, workspace,
                            s);
}
