// cellsum.cuh — scatter of a CTA's particles into the grid, summed per cell.
//
// The particle kernels of the sorted path end with a scatter of 27 node
// contributions per particle. Lanes first leave the terms of their particle in
// shared memory; then the CTA's threads share out (group, stencil row) items,
// where a group is the particles of one warp that have the same base cell: a
// thread walks the particles of its group, sums the three nodes of its row in
// registers and issues one 16-byte reduction per node. Against summing over
// lanes with shuffles (two rounds per node and component, 82 instructions per
// particle and node with the address arithmetic) a particle costs about 60
// instructions per row of three nodes, and a cell's particles take one
// reduction per node however many they are. The groups are found by matching
// cell keys over the warp, not by runs of equal neighbours, so particles that
// have crossed a cell border since the last sort still share their sums.
#pragma once
#include "pairs.cuh"
#include "substep.cuh"

namespace empm {

// ---- the scatter ------------------------------------------------------------
// Longest group: longer ones are cut, so that a crowded cell does not leave a
// CTA with few long sums.
constexpr int kCellGroupMax = 8;

// One particle's node contributions are
//   w (a + i B0 + j B1 + k B2) + dwx S0 + dwy S1 + dwz S2,   w = wx wy wz,
// for the momentum with a and B already multiplied by the particle's mass, S
// symmetric and w m as fourth component (MASS); or for an adjoint without a
// fourth component. A thread leaves the terms of its particle in two parts, the
// second one later (the stress is known last), so that the first need not stay
// in registers meanwhile. The particles of a group lie next to each other.
template <bool MASS, int NT>
struct CellScatter {
    float4 q[6][NT];                 // layout: cell_scatter_get
    int4   group[NT];                // first slot | length << 16, packed base node, first grid block, blocks per axis
    int    count[kCellGroupMax];     // groups by length - 1
};

// The kernel's first statement on its shared memory.
template <bool MASS, int NT>
__device__ __forceinline__ void cell_scatter_begin(CellScatter<MASS, NT>& sh) {
    if (threadIdx.x < kCellGroupMax) sh.count[threadIdx.x] = 0;
    __syncthreads();
}

// A thread's particle between the two parts.
struct CellSlot {
    int slot;        // where its terms are
    int length;      // of the group it heads, 0: it heads none
    int rank;        // of that group among those of its length
    int base;        // packed base node; -1: no particle, or not inside the grid
    int boff, NB;
};

// Groups of equal cells over the warp; every thread of the CTA takes part.
// valid: the thread has a particle, with base node b (unclamped) in an instance's grid of
// resolution G.
template <bool MASS, int NT>
__device__ __forceinline__ CellSlot cell_scatter_slot(CellScatter<MASS, NT>& sh, bool valid, const int b[3], int G,
                                                      int NB, int boff) {
    const int lane = threadIdx.x & 31;
    CellSlot c;
    c.boff = boff;
    c.NB = NB;
    c.base = -1;
    unsigned key = 0xffffffffu;
    if (valid && axis_in_grid(b[0], G) && axis_in_grid(b[1], G) && axis_in_grid(b[2], G)) {
        key = ((unsigned)(boff + block_of(b[0], b[1], b[2], NB)) << 6) | ((b[0] & 3) << 4) | ((b[1] & 3) << 2) |
              (b[2] & 3);
        c.base = (b[0] << 20) | (b[1] << 10) | b[2];
    }
    const unsigned peers = __match_any_sync(0xffffffffu, key);
    const int size = __popc(peers), rank = __popc(peers & ((1u << lane) - 1u));
    // slots: groups in the order of their first lanes
    int scan = rank == 0 ? size : 0;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const int up = __shfl_up_sync(0xffffffffu, scan, d);
        if (lane >= d) scan += up;
    }
    const int first = __shfl_sync(0xffffffffu, scan, __ffs(peers) - 1) - size;
    c.slot = (threadIdx.x & ~31) + first + rank;
    const bool head = c.base >= 0 && (rank & (kCellGroupMax - 1)) == 0;
    c.length = head ? min(kCellGroupMax, size - rank) : 0;
    c.rank = head ? atomicAdd(&sh.count[c.length - 1], 1) : 0;
    __syncwarp();   // the lanes have read what was fetched ahead into the places of the terms
    return c;
}

// First part.
template <bool MASS, int NT>
__device__ __forceinline__ void cell_scatter_put(CellScatter<MASS, NT>& sh, int slot, const float fx[3], float m,
                                                 V3 a, const M3& B) {
    if (MASS) {
        // the weights in z of the three nodes (wz1 = 1 - wz0 - wz2) and fz - 1.5
        float w0, w2, u0, u2;
        bspline_at(fx[2], 0, w0, u0);
        bspline_at(fx[2], 2, w2, u2);
        sh.q[0][slot] = make_float4(fx[0], fx[1], m, B.m[6]);
        sh.q[1][slot] = make_float4(w0, w2, u0, B.m[7]);
        sh.q[2][slot] = make_float4(a.x, a.y, a.z, B.m[8]);
        sh.q[3][slot] = make_float4(B.m[0], B.m[3], B.m[1], B.m[4]);
        float* q4 = reinterpret_cast<float*>(&sh.q[4][slot]);
        q4[0] = B.m[2];
        q4[1] = B.m[5];
    } else {
        float* q0 = reinterpret_cast<float*>(&sh.q[0][slot]);
        q0[0] = fx[0]; q0[1] = fx[1]; q0[2] = fx[2];
        sh.q[1][slot] = make_float4(a.x, a.y, a.z, B.m[6]);
        sh.q[2][slot] = make_float4(B.m[0], B.m[3], B.m[1], B.m[4]);
        sh.q[3][slot] = make_float4(B.m[2], B.m[5], B.m[7], B.m[8]);
    }
}

// Second part: S (MASS: symmetric).
template <bool MASS, int NT>
__device__ __forceinline__ void cell_scatter_put(CellScatter<MASS, NT>& sh, int slot, const M3& S) {
    if (MASS) {
        float* q4 = reinterpret_cast<float*>(&sh.q[4][slot]);
        q4[2] = S.m[0];
        q4[3] = S.m[8];
        sh.q[5][slot] = make_float4(S.m[1], S.m[4], S.m[2], S.m[5]);
    } else {
        reinterpret_cast<float*>(&sh.q[0][slot])[3] = S.m[7];
        sh.q[4][slot] = make_float4(S.m[1], S.m[4], S.m[2], S.m[5]);
        sh.q[5][slot] = make_float4(S.m[0], S.m[3], S.m[6], S.m[8]);
    }
}

struct CellTerms {
    float fx, fy, m;
    float w[3], u[3];   // weights and derivatives in z
    P3 a, B0, B1, B2, S0, S1, S2;
};

template <bool MASS, int NT>
__device__ __forceinline__ CellTerms cell_scatter_get(const CellScatter<MASS, NT>& sh, int p) {
    const float4 q0 = sh.q[0][p], q1 = sh.q[1][p], q2 = sh.q[2][p], q3 = sh.q[3][p], q4 = sh.q[4][p],
                 q5 = sh.q[5][p];
    CellTerms c;
    c.fx = q0.x; c.fy = q0.y;
    if (MASS) {
        c.m = q0.z;
        c.w[0] = q1.x; c.w[1] = (1.f - q1.x) - q1.y; c.w[2] = q1.y;
        c.u[0] = q1.z; c.u[1] = -2.f * q1.z - 1.f; c.u[2] = q1.z + 1.f;
        c.a = p3(f2_make(q2.x, q2.y), q2.z);
        c.B0 = p3(f2_make(q3.x, q3.y), q0.w);
        c.B1 = p3(f2_make(q3.z, q3.w), q1.w);
        c.B2 = p3(f2_make(q4.x, q4.y), q2.w);
        c.S0 = p3(f2_make(q4.z, q5.x), q5.z);
        c.S1 = p3(f2_make(q5.x, q5.y), q5.w);
        c.S2 = p3(f2_make(q5.z, q5.w), q4.w);
    } else {
        c.m = 0.f;
#pragma unroll
        for (int k = 0; k < 3; ++k) bspline_at(q0.z, k, c.w[k], c.u[k]);
        c.a = p3(f2_make(q1.x, q1.y), q1.z);
        c.B0 = p3(f2_make(q2.x, q2.y), q1.w);
        c.B1 = p3(f2_make(q2.z, q2.w), q3.z);
        c.B2 = p3(f2_make(q3.x, q3.y), q3.w);
        c.S0 = p3(f2_make(q5.x, q5.y), q5.z);
        c.S1 = p3(f2_make(q4.x, q4.y), q0.w);
        c.S2 = p3(f2_make(q4.z, q4.w), q5.w);
    }
    return c;
}

// A particle whose stencil leaves the grid (an initial state outside the
// band): its own thread writes the nodes that exist.
template <bool MASS, int NT>
__device__ __noinline__ void cell_scatter_edge(const CellScatter<MASS, NT>* sh, int slot, int bx, int by, int bz,
                                               int G, int NB, int boff, float4* grid, unsigned char* flags) {
    const CellTerms c = cell_scatter_get(*sh, slot);
    for (int n = 0; n < 27; ++n) {
        const int i = n / 9, j = (n / 3) % 3, k = n % 3;
        const int ix = base_clamp(bx) + i, iy = base_clamp(by) + j, iz = base_clamp(bz) + k;
        if (ix < 0 || iy < 0 || iz < 0 || ix >= G || iy >= G || iz >= G) continue;
        float wx, wy, ux, uy;
        bspline_at(c.fx, i, wx, ux);
        bspline_at(c.fy, j, wy, uy);
        const float wz = k == 0 ? c.w[0] : (k == 1 ? c.w[1] : c.w[2]);
        const float uz = k == 0 ? c.u[0] : (k == 1 ? c.u[1] : c.u[2]);
        P3 v = p3_mul(f2_both(wx * wy * wz), p3_fma(f2_both((float)k), c.B2,
                                                    p3_fma(f2_both((float)j), c.B1,
                                                           p3_fma(f2_both((float)i), c.B0, c.a))));
        v = p3_fma(f2_both(ux * wy * wz), c.S0, v);
        v = p3_fma(f2_both(wx * uy * wz), c.S1, v);
        v = p3_fma(f2_both(wx * wy * uz), c.S2, v);
        float x, y;
        f2_split(v.xy, x, y);
        const int blk = boff + block_of(ix, iy, iz, NB);
        red_add_v4(grid + (((long long)blk << 6) | ((ix & 3) << 4) | ((iy & 3) << 2) | (iz & 3)),
                   make_float4(x, y, v.z, MASS ? wx * wy * wz * c.m : 0.f));
        if (flags) flags[blk] = 1;
    }
}

// Sums and reductions, once both parts of all terms have been put. A work item
// is a group and the three stencil rows of one j: their 36 sums stay in
// registers, and the particle's terms, weights in y and z and a + j B1 are formed
// once for the three. With an item per row (a third of the registers, more warps)
// the fused kernel took 445 us on the 3.17M-particle population, with three 382.
// flags (may be NULL): the touched 4^3 blocks are marked.
template <bool MASS, int NT>
__device__ __forceinline__ void cell_scatter(CellScatter<MASS, NT>& sh, const CellSlot& c, float4* grid,
                                             unsigned char* flags) {
    __syncthreads();
    // groups in order of length, longest first: the threads of a warp then walk
    // groups of about the same length
    int total = 0, before = 0;
#pragma unroll
    for (int l = kCellGroupMax - 1; l >= 0; --l) {
        const int n = sh.count[l];
        if (l >= c.length) before += n;
        total += n;
    }
    if (c.length) sh.group[before + c.rank] = make_int4(c.slot | (c.length << 16), c.base, c.boff, c.NB);
    __syncthreads();
    const int items = 3 * total;
    for (int it = threadIdx.x; it < items; it += NT) {
        const int g = it / 3, j = it - 3 * g;
        const int4 gi = sh.group[g];
        P3 n[3][3];
        float w[3][3];
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
            for (int k = 0; k < 3; ++k) { n[i][k] = p3_zero(); w[i][k] = 0.f; }
        int p = gi.x & 0xffff;
        const int end = p + (gi.x >> 16);
        // weight in y at this j, as bspline_at forms it: s t t + k with t = fy - c
        const F2 fj = f2_both((float)j);
        const float cy = 1.5f - 0.5f * j, sy = j == 1 ? -1.f : 0.5f, ky = j == 1 ? 0.75f : 0.f;
#pragma unroll 1
        for (; p < end; ++p) {
            const CellTerms c = cell_scatter_get(sh, p);
            const float ty = c.fy - cy, sty = sy * ty;
            const float wy = sty * ty + ky, uy = sty + sty;
            const P3 aj = p3_fma(fj, c.B1, c.a);
#pragma unroll
            for (int i = 0; i < 3; ++i) {
                float wx, ux;
                bspline_at(c.fx, i, wx, ux);
                const float wxys = wx * wy;
                const F2 wxy = f2_both(wxys);
                // row terms: node k is wz_k (P + k Q) + dwz_k R
                const P3 a = i ? p3_fma(f2_both((float)i), c.B0, aj) : aj;
                const P3 P = p3_fma(f2_both(wx * uy), c.S1, p3_fma(f2_both(ux * wy), c.S0, p3_mul(wxy, a)));
                const P3 Q = p3_mul(wxy, c.B2), R = p3_mul(wxy, c.S2);
                const P3 PQ = p3_add(P, Q), PQQ = p3_add(PQ, Q);
                n[i][0] = p3_fma(f2_both(c.u[0]), R, p3_fma(f2_both(c.w[0]), P, n[i][0]));
                n[i][1] = p3_fma(f2_both(c.u[1]), R, p3_fma(f2_both(c.w[1]), PQ, n[i][1]));
                n[i][2] = p3_fma(f2_both(c.u[2]), R, p3_fma(f2_both(c.w[2]), PQQ, n[i][2]));
                if (MASS) {
                    const float ms = wxys * c.m;
#pragma unroll
                    for (int k = 0; k < 3; ++k) w[i][k] = fmaf(c.w[k], ms, w[i][k]);
                }
            }
        }
        const int NBg = gi.w;
        const int iy = ((gi.y >> 10) & 1023) + j, iz = gi.y & 1023;
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            const int ix = (gi.y >> 20) + i;
            const int rowblk = gi.z + ((ix >> 2) * NBg + (iy >> 2)) * NBg;
            const unsigned rowoff = ((ix & 3) << 4) | ((iy & 3) << 2);
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                float x, y;
                f2_split(n[i][k].xy, x, y);
                red_add_v4(grid + (((unsigned)(rowblk + ((iz + k) >> 2)) << 6) | rowoff | ((iz + k) & 3)),
                           make_float4(x, y, n[i][k].z, w[i][k]));
            }
            // the stencil's blocks are those of its corner rows
            if (flags && i != 1 && j != 1) {
                flags[rowblk + (iz >> 2)] = 1;
                flags[rowblk + ((iz + 2) >> 2)] = 1;
            }
        }
    }
}

}  // namespace empm
