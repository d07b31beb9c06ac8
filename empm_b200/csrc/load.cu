// load.cu — particle state between the caller's layout and the library's: instances of
// a batch (re)loaded from their specs in one launch, matrices as rows.
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/empm_b200.h"
#include "ctx.hpp"
#include "mat3.cuh"

using namespace empm;

namespace {

struct LoadTargets {
    float4*  x;
    float4*  v;
    F9Planes C, F;
    float *vol, *density, *E, *nu, *ys;
};

// Rows [first, first + count) of an instance per blockIdx.x. Reads each scalar array
// once and writes the state once: 3.2 M particles 470 MB. A batch of 12 bodies of 2 k
// particles took 160 copies and fills of slices instead, 2.3 ms of the host.
__global__ void __launch_bounds__(256) k_load_instances(const EmpmInstanceArrays* table, const LoadTargets out) {
    const EmpmInstanceArrays a = table[blockIdx.x];
    for (int i = blockIdx.y * blockDim.x + threadIdx.x; i < a.count; i += gridDim.y * blockDim.x) {
        const size_t p = (size_t)a.first + i;
        const auto scalar = [&](const float* src, int bit) {
            return src ? __ldg(src + ((a.broadcast >> bit) & 1 ? 0 : i)) : 0.f;
        };
        const auto vec = [&](const float* src, int bit) {
            if (!src) return make_float4(0.f, 0.f, 0.f, 0.f);
            src += (a.broadcast >> bit) & 1 ? 0 : 3 * (size_t)i;
            return make_float4(__ldg(src), __ldg(src + 1), __ldg(src + 2), 0.f);
        };
        float4 x = vec(a.x, 0);
        x.w = out.x[p].w;      // the mass lane is prepared from density and volume
        out.x[p] = x;
        out.v[p] = vec(a.v, 1);
        out.vol[p] = scalar(a.vol, 2);
        out.density[p] = scalar(a.density, 3);
        out.E[p] = scalar(a.E, 4);
        out.nu[p] = scalar(a.nu, 5);
        out.ys[p] = scalar(a.yield_stress, 6);
        f9_store(out.C, p, m3_zero());
        f9_store(out.F, p, m3_identity());
    }
}

// Matrix planes to rows of 9: loads of 16 B, rows gathered in shared memory (stride 9:
// no bank conflicts), stores of 16 B. Bound by its 72 B per particle; 500k particles
// 6.8 us against 17.2 us of a concatenation of the three planes.
constexpr int kRowThreads = 128;
__global__ void __launch_bounds__(kRowThreads) k_matrix_rows(const F9Planes planes, float4* out, int n) {
    __shared__ __align__(16) float rows[kRowThreads * 9];
    const int p0 = blockIdx.x * kRowThreads, p = p0 + threadIdx.x;
    if (p < n) {
        const M3 m = f9_load(planes, p);
#pragma unroll
        for (int k = 0; k < 9; ++k) rows[9 * threadIdx.x + k] = m.m[k];
    }
    __syncthreads();
    const int words = 9 * min(kRowThreads, n - p0);
    const size_t base = (size_t)p0 * 9;
    for (int i = threadIdx.x; 4 * i < words; i += kRowThreads) {
        if (4 * i + 4 <= words) {
            out[base / 4 + i] = *reinterpret_cast<const float4*>(rows + 4 * i);
        } else {
            for (int k = 4 * i; k < words; ++k) reinterpret_cast<float*>(out)[base + k] = rows[k];
        }
    }
}

}  // namespace

extern "C" int empm_matrix_rows(const float* planes, int n, float* out, void* stream) {
    if (n < 0 || (n && (!planes || !out)) || (((uintptr_t)planes | (uintptr_t)out) & 15))
        return empm_set_error(nullptr, EMPM_ERR_INVALID, "matrix rows: bad arguments (16-byte alignment needed)");
    if (n == 0) return EMPM_OK;
    k_matrix_rows<<<(n + kRowThreads - 1) / kRowThreads, kRowThreads, 0, (cudaStream_t)stream>>>(
        f9_planes(const_cast<float*>(planes), n), reinterpret_cast<float4*>(out), n);
    return empm_check_cuda(nullptr, cudaGetLastError(), "k_matrix_rows");
}

extern "C" int empm_load_instances(const EmpmInstanceArrays* table, int n_instances, int max_count, int n_total,
                                   EmpmParticles* out, float* vol, float* density, float* E, float* nu,
                                   float* yield_stress, void* stream) {
    if (n_instances < 0 || max_count < 0 || n_total < 0 || !out ||
        (n_instances && max_count && (!table || !out->x || !out->v || !out->C || !out->F || !vol || !density || !E || !nu ||
                                      !yield_stress)))
        return empm_set_error(nullptr, EMPM_ERR_INVALID, "load: bad arguments");
    if (n_instances == 0 || max_count == 0) return EMPM_OK;
    LoadTargets t;
    t.x = reinterpret_cast<float4*>(out->x);
    t.v = reinterpret_cast<float4*>(out->v);
    t.C = f9_planes(out->C, n_total);
    t.F = f9_planes(out->F, n_total);
    t.vol = vol; t.density = density; t.E = E; t.nu = nu; t.ys = yield_stress;
    const int g = (max_count + 255) / 256;
    k_load_instances<<<dim3(n_instances, g < 1024 ? g : 1024), 256, 0, (cudaStream_t)stream>>>(table, t);
    return empm_check_cuda(nullptr, cudaGetLastError(), "k_load_instances");
}
