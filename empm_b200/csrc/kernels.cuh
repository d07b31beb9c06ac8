// kernels.cuh — __global__ kernels of one MLS-MPM substep over a batch of
// independent simulation instances (a single simulation is a batch of one).
//
// Batch layout: the particles of instance i occupy [poff_i, poff_i + n_i) of
// every particle array, both in the caller's order and in the library's
// cell-sorted order (the sort key starts with the instance's grid blocks, so
// a sort never moves a particle across instances); the grids are the
// instances' blocked grids one after the other, instance i starting at the
// global 4^3 block boff_i. Every kernel looks its instance up in a small
// device table by particle index or block index.
//
// Launch paths:
//   * direct: one particle per thread, 16-byte vector reductions into the grid;
//   * sorted (rollouts): particles in cell order, re-sorted every few substeps;
//     P2G sums the contributions of same-cell particles of a warp and issues one
//     reduction per cell and node (default, cellsum.cuh), or accumulates per
//     chunk in a shared-memory node tile (option);
//     G2P gathers directly or from a staged shared-memory tile (option);
//   * the grid update visits only the 4^3 node blocks that P2G touched.
#pragma once
#include <limits.h>
#include "../../include/empm_b200.h"
#include "grid.cuh"
#include "substep.cuh"
#include "cellsum.cuh"

// Threads per CTA of the particle kernels that scatter per cell, and the
// minimum resident CTAs per SM asked of the compiler: for stress + P2G (at 5: 96
// registers, 46 us for 500k particles; at 4 51 us), with the G2P before it (at 4:
// 128 registers, no spills, 64.5 us and 371 us on the population; at 5 68.5 and
// 379 us, at 6 72 and 390 us; CTAs of 256 threads 5-10 % slower), and for G2P alone
// (CTAs of 128).
#ifndef EMPM_CELL_THREADS
#define EMPM_CELL_THREADS 128
#endif
#ifndef EMPM_P2G_MIN_CTAS
#define EMPM_P2G_MIN_CTAS 5
#endif
#ifndef EMPM_FUSED_MIN_CTAS
#define EMPM_FUSED_MIN_CTAS 4
#endif
#ifndef EMPM_G2P_MIN_CTAS
#define EMPM_G2P_MIN_CTAS 8
#endif

namespace empm {

// -------------------------------------------------------------------------
// instance table and per-launch context
// -------------------------------------------------------------------------
struct InstanceConsts {
    int   n, poff;            // particles
    int   G, NB, boff;        // grid: resolution, blocks per axis, first global block
    float dx, inv_dx, grid_lim, rpic, damping;
    float g[3];
    MaterialScalars ms;
};

struct Launch {
    const InstanceConsts* inst;
    int             n_inst;
    int             n_total;       // particles over all instances
    int             nblocks;       // grid blocks over all instances
    const EmpmStep* steps;         // device step tables: steps[table * n_inst + instance]
    int             table;         // step table of this substep
    unsigned*       status;
};

// per-instance view used by the particle/node device functions
struct StepConsts {
    int   G, NB, boff;
    float dx, inv_dx, grid_lim, rpic;
    // the material constants stay in the instance table: the return maps read
    // them only when a particle yields, so they are not held in registers
    // across a particle's substep (fused population kernel 560 -> 558 us)
    const MaterialScalars* ms;
    const EmpmStep* step;
    unsigned* status;
};

__device__ __forceinline__ int find_instance_particle(const Launch& L, int p) {
    int lo = 0, hi = L.n_inst - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (__ldg(&L.inst[mid].poff) <= p) lo = mid; else hi = mid - 1;
    }
    return lo;
}

__device__ __forceinline__ int find_instance_block(const Launch& L, int b) {
    int lo = 0, hi = L.n_inst - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (__ldg(&L.inst[mid].boff) <= b) lo = mid; else hi = mid - 1;
    }
    return lo;
}

__device__ __forceinline__ StepConsts consts_of(const Launch& L, int i) {
    const InstanceConsts* I = L.inst + i;
    StepConsts c;
    c.G = __ldg(&I->G);
    c.NB = __ldg(&I->NB);
    c.boff = __ldg(&I->boff);
    c.dx = __ldg(&I->dx);
    c.inv_dx = __ldg(&I->inv_dx);
    c.grid_lim = __ldg(&I->grid_lim);
    c.rpic = __ldg(&I->rpic);
    c.ms = &I->ms;
    c.step = L.steps + (size_t)L.table * L.n_inst + i;
    c.status = L.status;
    return c;
}

__device__ __forceinline__ long long gaddr(const StepConsts& c, int i, int j, int k) {
    return ((long long)(c.boff + block_of(i, j, k, c.NB)) << 6) | ((i & 3) << 4) | ((j & 3) << 2) | (k & 3);
}

// Addresses of the 27 nodes of a stencil with base node b: gaddr of node
// b + (i, j, k) is x(i) + y[j] + z[k]. The block index sits above the 6 bits of
// the local index, so gaddr's OR is a sum of one term per axis; x(i) carries
// the instance's block offset. Valid only for nodes inside the grid.
struct StencilAddr {
    int bx, boff, nb2;   // x[i] is rebuilt from these where it is used (fewer live registers)
    int y[3], z[3];
    EMPM_HD long long x(int i) const {
        const int ix = bx + i;
        return ((long long)(boff + (ix >> 2) * nb2) << 6) | ((ix & 3) << 4);
    }
    EMPM_HD long long at(int i, int j, int k) const { return x(i) + (long long)(y[j] + z[k]); }
};

EMPM_HD StencilAddr stencil_addr(int boff, int NB, const int b[3]) {
    StencilAddr a;
    a.bx = b[0];
    a.boff = boff;
    a.nb2 = NB * NB;
#pragma unroll
    for (int o = 0; o < 3; ++o) {
        const int iy = b[1] + o, iz = b[2] + o;
        a.y[o] = (((iy >> 2) * NB) << 6) | ((iy & 3) << 2);
        a.z[o] = ((iz >> 2) << 6) | (iz & 3);
    }
    return a;
}

// stencil node (i, j, k) inside the instance's grid (for stencils that are not entirely inside)
EMPM_HD bool node_in_grid(const int b[3], int i, int j, int k, int G) {
    return (unsigned)b[0] + i < (unsigned)G && (unsigned)b[1] + j < (unsigned)G && (unsigned)b[2] + k < (unsigned)G;
}

// -------------------------------------------------------------------------
// particle arrays
// -------------------------------------------------------------------------
struct ParticleArrays {
    float4*  x;      // (x, y, z, mass)
    float4*  v;      // (vx, vy, vz, 0)
    F9Planes C;
    F9Planes F;      // F_trial
};

struct MaterialArrays {
    const float* vol;
    float*       mu;
    float*       lam;
    float*       ys;
    const int*   sel;   // NULL = all simulated
    const int*   pid;   // caller index of each particle (NULL = identity)
};

// Stress + everything P2G needs for particle p (modifiers applied, material
// write-back, elastic F handed to G2P). Returns false for unsimulated particles.
template <int MAT = -1>
__device__ __forceinline__ bool prepare_particle(const ParticleArrays& P, const MaterialArrays& M, F9Planes Fe,
                                                 const StepConsts& c, int p, P2GParticle& q) {
    if (M.sel && __ldg(M.sel + p) != 0) return false;
    const EmpmStep& st = *c.step;
    if (st.hold) return false;   // held instance: no contribution this substep
    const float4 xm = __ldg(P.x + p);
    const float4 vv = __ldg(P.v + p);
    const V3 x = v3(xm.x, xm.y, xm.z);
    V3 v = v3(vv.x, vv.y, vv.z);
    if (st.n_modifiers > 0) {
        const int mi = M.pid ? __ldg(M.pid + p) : p;
        if (apply_modifiers(st, mi, x, xm.w, v)) P.v[p] = make_float4(v.x, v.y, v.z, vv.w);
    }
    float mu = __ldg(M.mu + p), lam = __ldg(M.lam + p), ys = __ldg(M.ys + p);
    const ConstitutiveOut co = constitutive_general<MAT>(f9_load(P.F, p), mu, lam, ys, st.dt, *c.ms);
    f9_store(Fe, p, co.F);
    if (co.mat_changed) { M.mu[p] = mu; M.lam[p] = lam; M.ys[p] = ys; }
    q.st = make_stencil(x, c.inv_dx);
    q.wm_scale = xm.w;
    q.v = v;
    q.Cd = damp_affine(f9_load(P.C, p), c.rpic);
    q.Sv = (-__ldg(M.vol + p)) * co.tau;
    return true;
}

__device__ __forceinline__ void mark_stencil_blocks(unsigned char* flags, const Stencil& st, const StepConsts& c) {
    const int G = c.G;
    const int lo[3] = {max(st.b[0], 0), max(st.b[1], 0), max(st.b[2], 0)};
    const int hi[3] = {min(st.b[0], G - 3) + 2, min(st.b[1], G - 3) + 2, min(st.b[2], G - 3) + 2};
    for (int bi = lo[0] >> 2; bi <= hi[0] >> 2; ++bi)
        for (int bj = lo[1] >> 2; bj <= hi[1] >> 2; ++bj)
            for (int bk = lo[2] >> 2; bk <= hi[2] >> 2; ++bk) flags[c.boff + (bi * c.NB + bj) * c.NB + bk] = 1;
}

// direct scatter of one prepared particle into the blocked grid
__device__ __forceinline__ void scatter_global(const P2GParticle& q, const StepConsts& c, float4* grid,
                                               unsigned char* flags) {
    const int G = c.G;
    const bool in_grid = stencil_in_grid(q.st, G);
    if (!in_grid) atomicOr(c.status, EMPM_STATUS_OUT_OF_BAND);
    const P2GPre pre = p2g_pre(q, c.dx, c.inv_dx, c.step->dt);
    p2g_emit(pre, [&](int i, int j, int k, float4 v) {
        if (in_grid || node_in_grid(q.st.b, i, j, k, G))
            red_add_v4(grid + gaddr(c, q.st.b[0] + i, q.st.b[1] + j, q.st.b[2] + k), v);
    });
    mark_stencil_blocks(flags, q.st, c);
}

// -------------------------------------------------------------------------
// direct path
// -------------------------------------------------------------------------
__global__ void __launch_bounds__(128) k_p2g_direct(ParticleArrays P, MaterialArrays M, F9Planes Fe, Launch L,
                                                    float4* grid, unsigned char* flags) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= L.n_total) return;
    const StepConsts c = consts_of(L, find_instance_particle(L, p));
    P2GParticle q;
    if (!prepare_particle(P, M, Fe, c, p, q)) return;
    scatter_global(q, c, grid, flags);
}

// -------------------------------------------------------------------------
// grid update over touched 4^3 blocks (both paths)
// -------------------------------------------------------------------------
struct GridUpdateArgs {
    float4*        mom;      // accumulation; zeroed here for the next substep
    float4*        vel;      // node velocity after the boundary conditions (w = node mass)
    unsigned char* flags;    // touched blocks; cleared here
    Launch         L;
    // optional store slot of the touched blocks (stored segments): per block its
    // 64 node momenta, then its 64 node velocities; the list count (zero before)
    // and ids. Of more than store_cap blocks the others are only counted.
    float4*        store = nullptr;
    int*           store_list = nullptr;
    int            store_cap = 0;
};

// Calls f(block) for the touched blocks, a warp per call (all its lanes).
// Touched blocks are neighbours, so a warp looks at blocks far apart: the marks of
// its chunk c are those of blocks c, c + chunks, c + 2 chunks ..., as few per warp as
// the launch's warps allow, and neighbouring warps read neighbouring bytes. That
// spreads the work as a list of the touched blocks would, without the two launches
// that reset and fill one (3.0 us of the 20 us of a 20k-particle substep; a list
// written by the P2G kernels themselves took the population's 367 -> 445 us, for
// the marks they then have to read). clear: the marks are reset.
template <typename F>
__device__ __forceinline__ void for_touched_blocks(unsigned char* marks, const Launch& L, bool clear, F f) {
    const int lane = threadIdx.x & 31;
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, warps = (gridDim.x * blockDim.x) >> 5;
    const int per = min(32, (L.nblocks + warps - 1) / warps);
    const int chunks = (L.nblocks + per - 1) / per;
    for (int c = warp; c < chunks; c += warps) {
        const int b = c + lane * chunks;
        const bool on = lane < per && b < L.nblocks && marks[b] != 0;
        unsigned mask = __ballot_sync(0xffffffffu, on);
        if (mask == 0u) continue;
        if (on && clear) marks[b] = 0;
        while (mask) {
            const int j = __ffs(mask) - 1;
            mask &= mask - 1u;
            f(c + j * chunks);
        }
    }
}

// Grid update over the touched blocks, one warp per block and two nodes per lane:
// normalisation, gravity, damping and boundary conditions. The accumulation is
// cleared for the next substep; kKeep leaves it and the marks in place (the adjoint
// replays the boundary conditions from the accumulated momentum).
template <bool kKeep>
__global__ void __launch_bounds__(256) k_grid_update(const GridUpdateArgs a) {
    const int lane = threadIdx.x & 31;
    for_touched_blocks(a.flags, a.L, !kKeep, [&](int b) {
        const long long base = (long long)b << 6;
        const float4 m0 = a.mom[base + lane];   // on their way while the instance is looked up
        const float4 m1 = a.mom[base + lane + 32];
        const int inst = find_instance_block(a.L, b);
        int slot = 0;
        if (a.store) {
            if (lane == 0) slot = atomicAdd(a.store_list, 1);
            slot = __shfl_sync(0xffffffffu, slot, 0);
        }
        const bool save = a.store && slot < a.store_cap;
        const InstanceConsts* I = a.L.inst + inst;
        const EmpmStep& st = a.L.steps[(size_t)a.L.table * a.L.n_inst + inst];
        const V3 g = v3(__ldg(&I->g[0]), __ldg(&I->g[1]), __ldg(&I->g[2]));
        const float damping = __ldg(&I->damping);
        const float dt = st.dt;
        const int n_coll = st.n_colliders;
        const int G = __ldg(&I->G), NB = __ldg(&I->NB), boff = __ldg(&I->boff);
        const float dx = __ldg(&I->dx);
        if (!kKeep) {
            a.mom[base + lane] = make_float4(0.f, 0.f, 0.f, 0.f);
            a.mom[base + lane + 32] = make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int in_block = lane + 32 * h;
            const float4 m = h ? m1 : m0;
            V3 v = grid_velocity(m, dt, g, damping);
            if (n_coll > 0) {
                int i, j, k;
                node_coords(((long long)(b - boff) << 6) | in_block, NB, i, j, k);
                if (i < G && j < G && k < G) {
                    const long long dense = ((long long)i * G + j) * G + k;
                    apply_colliders(st, i, j, k, G, dx, dense, v);
                }
            }
            const float4 v4 = make_float4(v.x, v.y, v.z, m.w);
            a.vel[base + in_block] = v4;
            if (save) {
                a.store[(long long)slot * 128 + in_block] = m;
                a.store[(long long)slot * 128 + 64 + in_block] = v4;
            }
        }
        if (save && lane == 0) a.store_list[1 + slot] = b;
    });
}

// -------------------------------------------------------------------------
// G2P (shared by both paths through the fetch functor)
// -------------------------------------------------------------------------
template <typename Fetch>
__device__ __forceinline__ void g2p_particle(const ParticleArrays& P, F9Planes Fe, const MaterialArrays& M,
                                             const ParticleArrays& out, const StepConsts& c, int p, Fetch fetch) {
    if (M.sel && __ldg(M.sel + p) != 0) {
        __stcs(out.x + p, make_float4(0.f, 0.f, 0.f, __ldg(P.x + p).w));
        __stcs(out.v + p, make_float4(0.f, 0.f, 0.f, 0.f));
        f9_store(out.C, p, m3_zero());
        f9_store(out.F, p, m3_identity());
        return;
    }
    if (c.step->hold) {   // held instance: the state passes through unchanged
        __stcs(out.x + p, __ldg(P.x + p));
        __stcs(out.v + p, __ldg(P.v + p));
        f9_store(out.C, p, f9_load(P.C, p));
        f9_store(out.F, p, f9_load(P.F, p));
        return;
    }
    const float dt = c.step->dt;
    const float4 xm = __ldg(P.x + p);
    const V3 x = v3(xm.x, xm.y, xm.z);
    const Stencil st = make_stencil(x, c.inv_dx);
    const bool in_grid = stencil_in_grid(st, c.G);
    const G2POut o = g2p_gather(st, c.inv_dx, fetch.bind(st, in_grid));
    const float dx = 1.f / c.inv_dx;
    const float lo = dx * 2.f, hi = c.grid_lim - dx * 2.f;
    V3 nx = x + dt * o.v;
    nx = v3(fminf(fmaxf(nx.x, lo), hi), fminf(fmaxf(nx.y, lo), hi), fminf(fmaxf(nx.z, lo), hi));
    const M3 Fn = (m3_identity() + dt * o.gradv) * f9_load(Fe, p);
    __stcs(out.x + p, make_float4(nx.x, nx.y, nx.z, xm.w));
    __stcs(out.v + p, make_float4(o.v.x, o.v.y, o.v.z, 0.f));
    f9_store(out.C, p, o.C);
    f9_store(out.F, p, Fn);
    unsigned flags = 0;
    if (!finite3(o.v) || !finite3(nx) || !isfinite(Fn.m[0] + Fn.m[4] + Fn.m[8])) flags |= EMPM_STATUS_NAN;
    if (fmaxf(fmaxf(fabsf(o.v.x), fabsf(o.v.y)), fabsf(o.v.z)) * dt > dx) flags |= EMPM_STATUS_CFL;
    if (!in_grid) flags |= EMPM_STATUS_OUT_OF_BAND;
    if (flags) atomicOr(c.status, flags);
}

// Node velocities from the blocked grid. bind() precomputes the stencil's
// node addresses; nodes outside the grid read as zero.
struct GlobalFetch {
    const float4* vel;
    const StepConsts* c;
    struct Bound {
        const float4* vel;
        StencilAddr sa;
        const int* b;
        int G;
        bool in_grid;
        __device__ __forceinline__ V3 operator()(int i, int j, int k) const {
            if (!in_grid && !node_in_grid(b, i, j, k, G)) return v3(0.f, 0.f, 0.f);
            const float4 g = __ldg(vel + sa.at(i, j, k));
            return v3(g.x, g.y, g.z);
        }
    };
    __device__ __forceinline__ Bound bind(const Stencil& st, bool in_grid) const {
        return Bound{vel, stencil_addr(c->boff, c->NB, st.b), st.b, c->G, in_grid};
    }
};

// G2P gather of a stencil inside the grid, factorised over the inner axis: per
// row (i, j) the three nodes are combined with wz, dwz and k wz first, then the
// rows with weights in x and y; x and y components travel as pairs.
__device__ __forceinline__ G2POut g2p_gather_rows(const int b[3], const float fx[3], float inv_dx, int boff, int NB,
                                                  const float4* __restrict__ vel) {
    P3 V = p3_zero(), M0 = V, M1 = V, M2 = V;   // sum wg, and its moments in i, j, k
    P3 g0 = V, g1 = V, g2 = V;                  // columns of sum grid_v (x) dweight / inv_dx
    F2 wz[3], uz[3];
    unsigned zpart[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        float w, u;
        bspline_at(fx[2], k, w, u);
        wz[k] = f2_both(w);
        uz[k] = f2_both(u);
        zpart[k] = ((unsigned)((b[2] + k) >> 2) << 6) | ((b[2] + k) & 3);
    }
    const F2 kz2 = f2_add(wz[2], wz[2]);
#pragma unroll 1
    for (int i = 0; i < 3; ++i) {
        float wx, ux;
        bspline_at(fx[0], i, wx, ux);
        const int ix = b[0] + i;
        const int xblk = boff + (ix >> 2) * NB * NB;
        const unsigned xoff = (ix & 3) << 4;
        P3 Vi = p3_zero();
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            const int iy = b[1] + j;
            const unsigned row = ((unsigned)(xblk + (iy >> 2) * NB) << 6) + (xoff | ((iy & 3) << 2));
            const float4 a0 = __ldg(vel + (row + zpart[0])), a1 = __ldg(vel + (row + zpart[1])),
                         a2 = __ldg(vel + (row + zpart[2]));
            const P3 n0 = p3(f2_make(a0.x, a0.y), a0.z), n1 = p3(f2_make(a1.x, a1.y), a1.z),
                     n2 = p3(f2_make(a2.x, a2.y), a2.z);
            float wy, uy;
            bspline_at(fx[1], j, wy, uy);
            const F2 wxy = f2_both(wx * wy);
            const P3 T0 = p3_fma(wz[2], n2, p3_fma(wz[1], n1, p3_mul(wz[0], n0)));
            const P3 T1 = p3_fma(uz[2], n2, p3_fma(uz[1], n1, p3_mul(uz[0], n0)));
            const P3 Tk = p3_fma(kz2, n2, p3_mul(wz[1], n1));
            Vi = p3_fma(wxy, T0, Vi);
            if (j == 1) M1 = p3_fma(wxy, T0, M1);
            if (j == 2) M1 = p3_fma(f2_add(wxy, wxy), T0, M1);
            M2 = p3_fma(wxy, Tk, M2);
            g0 = p3_fma(f2_both(ux * wy), T0, g0);
            g1 = p3_fma(f2_both(wx * uy), T0, g1);
            g2 = p3_fma(wxy, T1, g2);
        }
        V = p3_add(V, Vi);
        M0 = p3_fma(f2_both((float)i), Vi, M0);
    }
    G2POut o;
    o.v.z = V.z;
    f2_split(V.xy, o.v.x, o.v.y);
    const P3 mc[3] = {M0, M1, M2}, gc[3] = {g0, g1, g2};
    const float c4 = 4.f * inv_dx;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        float x, y;
        f2_split(mc[c].xy, x, y);
        o.C.m[c] = c4 * (x - fx[c] * o.v.x);
        o.C.m[3 + c] = c4 * (y - fx[c] * o.v.y);
        o.C.m[6 + c] = c4 * (mc[c].z - fx[c] * o.v.z);
        f2_split(gc[c].xy, x, y);
        o.gradv.m[c] = inv_dx * x;
        o.gradv.m[3 + c] = inv_dx * y;
        o.gradv.m[6 + c] = inv_dx * gc[c].z;
    }
    return o;
}

// The same for a stencil that leaves the grid: nodes outside read as zero.
__device__ __noinline__ void g2p_gather_edge(G2POut* o, float x, float y, float z, float inv_dx, int boff, int NB,
                                             int G, const float4* vel) {
    const Stencil st = make_stencil(v3(x, y, z), inv_dx);
    const GlobalFetch::Bound fetch{vel, stencil_addr(boff, NB, st.b), st.b, G, false};
    *o = g2p_gather_rt(st, inv_dx, fetch);
}

// ---- fetching ahead ---------------------------------------------------------
// With 16 warps per SM the gather's waits are not hidden behind other warps, and
// the particle's F and material would be waited for once more after it. They are
// sent for before the gather, straight into the thread's part of the scatter's
// shared memory (cp.async), which is free until then (population fused kernel
// 397 -> 371 us; sending for the nodes of the warp's cells as well, to share them
// there: 362 us, but 66.3 against 64.5 us for 500k particles at 4 per cell).
__device__ __forceinline__ void copy_ahead16(void* dst, const void* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src));
}
__device__ __forceinline__ void copy_ahead4(void* dst, const void* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src));
}

struct Ahead { M3 F; float mu, lam, ys, vol; };

template <int NT>
__device__ __forceinline__ void particle_ahead(CellScatter<true, NT>& sh, const F9Planes& F, const MaterialArrays& M,
                                               int p) {
    const int t = threadIdx.x;
    copy_ahead16(&sh.q[0][t], F.a + p);
    copy_ahead16(&sh.q[1][t], F.b + p);
    copy_ahead4(&sh.q[2][t].x, F.c + p);
    copy_ahead4(&sh.q[2][t].y, M.mu + p);
    copy_ahead4(&sh.q[2][t].z, M.lam + p);
    copy_ahead4(&sh.q[2][t].w, M.ys + p);
    copy_ahead4(&sh.q[3][t].x, M.vol + p);
}

template <int NT>
__device__ __forceinline__ Ahead particle_arrived(const CellScatter<true, NT>& sh) {
    asm volatile("cp.async.wait_all;" ::: "memory");
    const int t = threadIdx.x;
    const float4 a = sh.q[0][t], b = sh.q[1][t], m = sh.q[2][t];
    Ahead r;
    r.F.m[0] = a.x; r.F.m[1] = a.y; r.F.m[2] = a.z; r.F.m[3] = a.w;
    r.F.m[4] = b.x; r.F.m[5] = b.y; r.F.m[6] = b.z; r.F.m[7] = b.w;
    r.F.m[8] = m.x;
    r.mu = m.y;
    r.lam = m.z;
    r.ys = m.w;
    r.vol = sh.q[3][t].x;
    return r;
}

// G2P of particle p at (x, mass) = xm: its gathered velocity and affine matrix
// are returned, nx is the clamped new position, Fn the new trial F and ah what was
// fetched ahead for it; status bits are set.
template <int NT>
__device__ __forceinline__ G2POut g2p_move(CellScatter<true, NT>& sh, const StepConsts& c, float dt, float4 xm,
                                           const F9Planes& Fe, const MaterialArrays& M, int p, const float4* vel,
                                           V3& nx, M3& Fn, Ahead& ah) {
    particle_ahead(sh, Fe, M, p);
    const float xs[3] = {xm.x, xm.y, xm.z};
    int b[3];
    float fx[3];
    bool in_grid = true;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        b[a] = base_unclamped(xs[a], c.inv_dx);
        fx[a] = base_frac(xs[a], c.inv_dx, b[a]);
        in_grid = in_grid && axis_in_grid(b[a], c.G);
    }
    G2POut o;
    if (in_grid) {
        o = g2p_gather_rows(b, fx, c.inv_dx, c.boff, c.NB, vel);
    } else {
        G2POut e;
        g2p_gather_edge(&e, xm.x, xm.y, xm.z, c.inv_dx, c.boff, c.NB, c.G, vel);
        o = e;
    }
    const float dx = 1.f / c.inv_dx;
    const float lo = dx * 2.f, hi = c.grid_lim - dx * 2.f;
    nx = v3(xm.x, xm.y, xm.z) + dt * o.v;
    nx = v3(fminf(fmaxf(nx.x, lo), hi), fminf(fmaxf(nx.y, lo), hi), fminf(fmaxf(nx.z, lo), hi));
    ah = particle_arrived(sh);
    Fn = (m3_identity() + dt * o.gradv) * ah.F;
    unsigned bad = 0;
    if (!finite3(o.v) || !finite3(nx) || !isfinite(Fn.m[0] + Fn.m[4] + Fn.m[8])) bad |= EMPM_STATUS_NAN;
    if (fmaxf(fmaxf(fabsf(o.v.x), fabsf(o.v.y)), fabsf(o.v.z)) * dt > dx) bad |= EMPM_STATUS_CFL;
    if (!in_grid) bad |= EMPM_STATUS_OUT_OF_BAND;
    if (bad) atomicOr(c.status, bad);
    return o;
}

__global__ void __launch_bounds__(128, EMPM_G2P_MIN_CTAS) k_g2p_direct(ParticleArrays P, F9Planes Fe, MaterialArrays M,
                                                    ParticleArrays out, Launch L, const float4* vel) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= L.n_total) return;
    const StepConsts c = consts_of(L, find_instance_particle(L, p));
    GlobalFetch f{vel, &c};
    g2p_particle(P, Fe, M, out, c, p, f);
}

// -------------------------------------------------------------------------
// sorted path: cell keys, counting sort, permutation
// -------------------------------------------------------------------------
// Sort key of a particle: its base cell in block-major order over the whole
// batch, ((boff + block) << 6) | in-block cell, so one counting sort orders
// particles by instance, 4^3 block and cell. Out-of-band cells are clamped.
__device__ __forceinline__ int cell_key(const InstanceConsts* I, float4 xm) {
    const int G = __ldg(&I->G), NB = __ldg(&I->NB);
    const float inv_dx = __ldg(&I->inv_dx);
    const float xs[3] = {xm.x, xm.y, xm.z};
    int b[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const int t = base_node(xs[a], inv_dx);
        b[a] = t < 0 ? 0 : (t >= G ? G - 1 : t);
    }
    const int blk = __ldg(&I->boff) + block_of(b[0], b[1], b[2], NB);
    return (blk << 6) | ((b[0] & 3) << 4) | ((b[1] & 3) << 2) | (b[2] & 3);
}

__global__ void k_sort_keys(const float4* x, Launch L, int* keys, int* ranks, int* cell_counts, int* block_counts) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= L.n_total) return;
    const int key = cell_key(L.inst + find_instance_particle(L, p), __ldg(x + p));
    const int blk = key >> 6;
    keys[p] = key;
    ranks[p] = atomicAdd(cell_counts + key, 1);
    atomicAdd(block_counts + blk, 1);
}

// number of chunks (<= `chunk` particles, never spanning two blocks) per block
__global__ void k_chunk_counts(const int* block_counts, int* chunk_counts, int nblocks, int chunk) {
    const int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= nblocks) return;
    chunk_counts[b] = (block_counts[b] + chunk - 1) / chunk;
}

// Cell offsets: one warp per block, exclusive scan of its 64 cell counts on
// top of the block's start offset; writes the block's chunks; zeroes the
// counts for the next sort. Empty blocks only report the chunk total.
__global__ void k_cell_scan(int* cell_counts, int* block_counts, const int* block_offsets, const int* chunk_offsets,
                            const int* chunk_counts, int* cell_offsets, int2* chunks, int* nchunks, int nblocks,
                            int chunk) {
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (warp >= nblocks) return;
    const int cnt = block_counts[warp];
    if (warp == nblocks - 1 && lane == 0) *nchunks = chunk_offsets[warp] + chunk_counts[warp];
    if (cnt == 0) return;
    const long long c0 = (long long)warp * 64 + 2 * lane;
    const int a = cell_counts[c0], b = cell_counts[c0 + 1];
    int incl = a + b;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, incl, d);
        if (lane >= d) incl += t;
    }
    const int off = block_offsets[warp];
    const int excl = incl - (a + b) + off;
    cell_offsets[c0] = excl;
    cell_offsets[c0 + 1] = excl + a;
    cell_counts[c0] = 0;
    cell_counts[c0 + 1] = 0;
    const int co = chunk_offsets[warp];
    for (int k = lane; k * chunk < cnt; k += 32) chunks[co + k] = make_int2(off + k * chunk, min(chunk, cnt - k * chunk));
    __syncwarp();
    if (lane == 0) block_counts[warp] = 0;
}

// -------------------------------------------------------------------------
// single substeps of many particles: the order of the cells
// -------------------------------------------------------------------------
// Puts the particles of a cell next to one another for one P2G, without moving
// their state: counts and ranks per cell, a range of the order per cell (cells come
// in any order, so a block's cells claim theirs with one atomic instead of a scan
// over the grid), the particles into the ranges. 500k particles in random order,
// 128^3 cells: 12.3 + 4.8 + 6.6 us; the first is bound by its returning atomics (43.7
// us while every particle marked its block, now the first of each cell does).
__global__ void k_order_count(const float4* x, Launch L, int2* keys, int* counts, unsigned char* marks, int* next) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p == 0) *next = 0;
    if (p >= L.n_total) return;
    const InstanceConsts* I = L.inst + find_instance_particle(L, p);
    const int key = cell_key(I, __ldg(x + p));
    const int rank = atomicAdd(counts + key, 1);
    if (rank == 0) marks[key >> 6] = 1;
    keys[p] = make_int2(key, rank);
}

__global__ void __launch_bounds__(256) k_order_ranges(Launch L, int* counts, int* offsets, unsigned char* marks,
                                                      int* next) {
    const int lane = threadIdx.x & 31;
    for_touched_blocks(marks, L, true, [&](int b) {
        const long long c0 = ((long long)b << 6) + 2 * lane;
        const int2 n = *reinterpret_cast<const int2*>(counts + c0);
        int incl = n.x + n.y;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int t = __shfl_up_sync(0xffffffffu, incl, d);
            if (lane >= d) incl += t;
        }
        int base = 0;
        if (lane == 31) base = atomicAdd(next, incl);
        const int first = __shfl_sync(0xffffffffu, base, 31) + incl - n.x - n.y;
        *reinterpret_cast<int2*>(offsets + c0) = make_int2(first, first + n.x);
        *reinterpret_cast<int2*>(counts + c0) = make_int2(0, 0);
    });
}

__global__ void k_order_fill(const int2* keys, const int* offsets, int* order, int n) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= n) return;
    const int2 k = __ldg(keys + p);
    order[__ldg(offsets + k.x) + k.y] = p;
}

struct PermuteArgs {
    ParticleArrays src, dst;
    const float* vol_s; float* vol_d;
    const float* mu_s;  float* mu_d;
    const float* lam_s; float* lam_d;
    const float* ys_s;  float* ys_d;
    const int*   sel_s; int*   sel_d;
    const int*   pid_s; int*   pid_d;   // pid_s NULL: source is in caller order
    F9Planes     fe_s, fe_d;             // elastic F (fe_s.a NULL: not moved)
    const int*   keys;
    const int*   ranks;
    const int*   offsets;    // cell offsets
    int n;
};

// src order -> sorted order: dst = cell_offsets[keys[p]] + ranks[p]
__global__ void k_sort_scatter(const PermuteArgs a) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= a.n) return;
    const int d = __ldg(a.offsets + __ldg(a.keys + p)) + __ldg(a.ranks + p);
    a.dst.x[d] = __ldg(a.src.x + p);
    a.dst.v[d] = __ldg(a.src.v + p);
    f9_store(a.dst.C, d, f9_load(a.src.C, p));
    f9_store(a.dst.F, d, f9_load(a.src.F, p));
    a.vol_d[d] = __ldg(a.vol_s + p);
    a.mu_d[d] = __ldg(a.mu_s + p);
    a.lam_d[d] = __ldg(a.lam_s + p);
    a.ys_d[d] = __ldg(a.ys_s + p);
    a.sel_d[d] = a.sel_s ? __ldg(a.sel_s + p) : 0;
    a.pid_d[d] = a.pid_s ? __ldg(a.pid_s + p) : p;
    if (a.fe_s.a) f9_store(a.fe_d, d, f9_load(a.fe_s, p));
}

struct UnsortArgs {
    ParticleArrays src, dst;      // sorted -> caller order
    F9Planes Fe_s, Fe_d;          // elastic F of the last substep
    const float* mu_s;  float* mu_d;
    const float* lam_s; float* lam_d;
    const float* ys_s;  float* ys_d;
    const int*   pid;
    int n;
};

__global__ void k_unsort(const UnsortArgs a) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= a.n) return;
    const int d = __ldg(a.pid + p);
    a.dst.x[d] = __ldg(a.src.x + p);
    a.dst.v[d] = __ldg(a.src.v + p);
    f9_store(a.dst.C, d, f9_load(a.src.C, p));
    f9_store(a.dst.F, d, f9_load(a.src.F, p));
    f9_store(a.Fe_d, d, f9_load(a.Fe_s, p));
    a.mu_d[d] = __ldg(a.mu_s + p);
    a.lam_d[d] = __ldg(a.lam_s + p);
    a.ys_d[d] = __ldg(a.ys_s + p);
}

// -------------------------------------------------------------------------
// sorted path, default P2G: contributions summed per cell (cellsum.cuh)
// -------------------------------------------------------------------------
// Stress and scatter of a CTA's particles; every thread takes part. A thread
// with valid set has particle p at x with velocity v, affine matrix C and trial F
// Ft: velocity modifiers, return map and stress are applied, the elastic F, the
// material scalars when they change and (v_out not NULL) the velocity after the
// modifiers are written, and the contributions
//   (weight * mass) (v + C dpos) - dt vol stress dweight, dpos = ((i, j, k) - fx) dx,
// go into the grid: a = v - dx C fx, B = dx C and S = -dt inv_dx vol stress.
// TAPE: for a tape, with the general constitutive update.
template <int MAT, bool TAPE, int NT>
__device__ __forceinline__ void p2g_cells(CellScatter<true, NT>& sh, bool valid, const StepConsts& c,
                                          const EmpmStep& sp, const MaterialArrays& M, int p, V3 x, float mass, V3 v,
                                          const M3& C, const M3& Ft, float mu, float lam, float ys, float vol,
                                          const F9Planes& Fe, float4* v_out, float4* grid, unsigned char* flags) {
    const float xs[3] = {x.x, x.y, x.z};
    int b[3] = {0, 0, 0};
    if (valid)
#pragma unroll
        for (int a = 0; a < 3; ++a) b[a] = base_unclamped(xs[a], c.inv_dx);
    const CellSlot cell = cell_scatter_slot(sh, valid, b, c.G, c.NB, c.boff);
    if (valid) {
        if (sp.n_modifiers > 0) {
            const int mi = M.pid ? __ldg(M.pid + p) : p;
            apply_modifiers(sp, mi, x, mass, v);
        }
        if (v_out) v_out[p] = make_float4(v.x, v.y, v.z, 0.f);
        float fx[3];
#pragma unroll
        for (int a = 0; a < 3; ++a) fx[a] = base_frac(xs[a], c.inv_dx, b[a]);
        const M3 B = (mass * c.dx) * damp_affine(C, c.rpic);
        cell_scatter_put(sh, cell.slot, fx, mass, mass * v - B * v3(fx[0], fx[1], fx[2]), B);
        const ConstitutiveOut co = TAPE ? constitutive_general<MAT>(Ft, mu, lam, ys, sp.dt, *c.ms)
                                        : constitutive<MAT>(Ft, mu, lam, ys, sp.dt, *c.ms);
        f9_store(Fe, p, co.F);
        if (co.mat_changed) { M.mu[p] = mu; M.lam[p] = lam; M.ys[p] = ys; }
        cell_scatter_put(sh, cell.slot, (sp.dt * c.inv_dx * -vol) * co.tau);
        if (cell.base < 0) {
            atomicOr(c.status, EMPM_STATUS_OUT_OF_BAND);
            cell_scatter_edge(&sh, cell.slot, b[0], b[1], b[2], c.G, c.NB, c.boff, grid, flags);
        }
    }
    cell_scatter(sh, cell, grid, flags);
}

// order: NULL for particles sorted by cell, else the order that makes them so (single
// substeps, k_order_*). Reading the state through it costs 15 sectors a particle: 500k
// in random order 74 us (jelly), 83 (sand), against 42 us sorted.
template <int NT, int MAT, int MINB, bool TAPE>
__global__ void __launch_bounds__(NT, MINB) k_p2g_cells(ParticleArrays P, MaterialArrays M, F9Planes Fe, Launch L,
                                                        float4* grid, unsigned char* flags, const int* order) {
    __shared__ CellScatter<true, NT> sh;
    cell_scatter_begin(sh);
    int p = blockIdx.x * NT + threadIdx.x;
    const bool in_range = p < L.n_total;
    if (order && in_range) p = __ldg(order + p);
    const StepConsts c = consts_of(L, in_range ? find_instance_particle(L, p) : 0);
    const EmpmStep& sp = *c.step;
    // a held instance contributes nothing this substep
    const bool valid = in_range && !(M.sel && __ldg(M.sel + p) != 0) && !sp.hold;
    float4 xm = make_float4(0.f, 0.f, 0.f, 0.f), vv = xm;
    M3 C = m3_zero(), F = C;
    float mu = 0.f, lam = 0.f, ys = 0.f, vol = 0.f;
    if (valid) {
        xm = __ldg(P.x + p);
        vv = __ldg(P.v + p);
        C = f9_load(P.C, p);
        F = f9_load(P.F, p);
        mu = __ldg(M.mu + p);
        lam = __ldg(M.lam + p);
        ys = __ldg(M.ys + p);
        vol = __ldg(M.vol + p);
    }
    p2g_cells<MAT, TAPE>(sh, valid, c, sp, M, p, v3(xm.x, xm.y, xm.z), xm.w, v3(vv.x, vv.y, vv.z), C, F, mu, lam, ys, vol,
                   Fe, sp.n_modifiers > 0 ? P.v : nullptr, grid, flags);
}

// -------------------------------------------------------------------------
// sorted path, fused: the G2P of substep s-1 and the stress + P2G of substep s
// in one pass over the particles
// -------------------------------------------------------------------------
// Between two such kernels a particle's persistent state is its position and
// its elastic F (plus the material scalars); its velocity, affine matrix and
// trial F are consumed by the P2G in the same thread, so they are not written
// back. Position and elastic F are updated in place: a thread reads and writes
// only its own particle. The grid velocities of substep s-1 (vel) are read,
// the accumulator of substep s (mom, cleared by the grid update of s-1) is
// written: the two are separate buffers. A run of fused substeps starts with
// the separate stress + P2G and ends with the separate G2P, which writes the
// full state. Held instances (step-table hold) must stay held once held within
// the run: when a particle's instance becomes held at substep s, its state
// after the G2P of s-1 is written in full, then left alone.
template <int NT, int MAT, int MINB, bool TAPE>
__global__ void __launch_bounds__(NT, MINB) k_g2p2g(ParticleArrays P, MaterialArrays M, F9Planes Fe, Launch L,
                                                    int g2p_table, const float4* vel, float4* mom,
                                                    unsigned char* flags) {
    __shared__ CellScatter<true, NT> sh;
    cell_scatter_begin(sh);
    const int p = blockIdx.x * NT + threadIdx.x;
    const int inst = p < L.n_total ? find_instance_particle(L, p) : 0;
    const StepConsts c = consts_of(L, inst);   // substep s: stress + P2G
    const EmpmStep& sg = L.steps[(size_t)g2p_table * L.n_inst + inst];   // substep s-1: G2P
    const EmpmStep& sp = *c.step;
    // lanes that run the G2P of substep s-1: simulated, not held
    bool valid = p < L.n_total && !(M.sel && __ldg(M.sel + p) != 0) && !sg.hold;
    const float4 xm = valid ? __ldg(P.x + p) : make_float4(0.f, 0.f, 0.f, 0.f);
    V3 nx;
    M3 Fn;
    Ahead ah;
    G2POut o;
    if (valid) {
        o = g2p_move(sh, c, sg.dt, xm, Fe, M, p, vel, nx, Fn, ah);
        P.x[p] = make_float4(nx.x, nx.y, nx.z, xm.w);
        if (sp.hold) {
            // held from substep s on: keep the state after this G2P
            valid = false;
            P.v[p] = make_float4(o.v.x, o.v.y, o.v.z, 0.f);
            f9_store(P.C, p, o.C);
            f9_store(P.F, p, Fn);
        }
    }
    p2g_cells<MAT, TAPE>(sh, valid, c, sp, M, p, nx, xm.w, o.v, o.C, Fn, ah.mu, ah.lam, ah.ys, ah.vol, Fe, nullptr, mom,
                   flags);
}

// Stored segments of a differentiable rollout (cell-sorted): the G2P of
// substep k-1 and the stress + P2G of substep k in one pass, writing what the
// reverse pass reads instead of handing state from kernel to kernel: the full
// state before substep k (its velocity after the modifiers, as the P2G of the
// separate kernels leaves it), the mu / lam / yield snapshot before substep k
// and the elastic F of substep k. Segments hold no instances (step-table hold)
// and their particles stay in one order, so every thread writes only its own
// particle of the substep-k arrays.
struct SegmentStoreArgs {
    ParticleArrays prev;     // state before substep k-1 (x read)
    F9Planes       fe_prev;  // elastic F of substep k-1
    ParticleArrays cur;      // out: state before substep k
    F9Planes       fe_cur;   // out: elastic F of substep k
    float*         snap;     // out: mu | lam | yield before substep k, stride np
    long long      np;
};

template <int NT, int MAT, int MINB, bool TAPE>
__global__ void __launch_bounds__(NT, MINB) k_g2p2g_store(MaterialArrays M, Launch L, int g2p_table,
                                                          const float4* vel, float4* mom, unsigned char* flags,
                                                          SegmentStoreArgs a) {
    __shared__ CellScatter<true, NT> sh;
    cell_scatter_begin(sh);
    const int p = blockIdx.x * NT + threadIdx.x;
    const int inst = p < L.n_total ? find_instance_particle(L, p) : 0;
    const StepConsts c = consts_of(L, inst);   // substep k: stress + P2G
    const bool valid = p < L.n_total && !(M.sel && __ldg(M.sel + p) != 0);
    const float4 xm = p < L.n_total ? __ldg(a.prev.x + p) : make_float4(0.f, 0.f, 0.f, 0.f);
    V3 nx;
    M3 Fn;
    Ahead ah;
    G2POut o;
    if (valid) {
        const float dt = L.steps[(size_t)g2p_table * L.n_inst + inst].dt;   // substep k-1
        o = g2p_move(sh, c, dt, xm, a.fe_prev, M, p, vel, nx, Fn, ah);
        a.snap[p] = ah.mu;
        a.snap[a.np + p] = ah.lam;
        a.snap[2 * a.np + p] = ah.ys;
        a.cur.x[p] = make_float4(nx.x, nx.y, nx.z, xm.w);
        f9_store(a.cur.C, p, o.C);
        f9_store(a.cur.F, p, Fn);
    } else if (p < L.n_total) {
        // unsimulated: the G2P writes the reference's constant state, no P2G
        a.snap[p] = __ldg(M.mu + p);
        a.snap[a.np + p] = __ldg(M.lam + p);
        a.snap[2 * a.np + p] = __ldg(M.ys + p);
        a.cur.x[p] = make_float4(0.f, 0.f, 0.f, xm.w);
        a.cur.v[p] = make_float4(0.f, 0.f, 0.f, 0.f);
        f9_store(a.cur.C, p, m3_zero());
        f9_store(a.cur.F, p, m3_identity());
    }
    p2g_cells<MAT, TAPE>(sh, valid, c, *c.step, M, p, nx, xm.w, o.v, o.C, Fn, ah.mu, ah.lam, ah.ys, ah.vol, a.fe_cur,
                   a.cur.v, mom, flags);
}

// Threads per CTA of the kernels above, and few: launches that would leave
// SMs idle at the usual size (particle_threads) take the small CTAs.
constexpr int kCellThreads = EMPM_CELL_THREADS;
constexpr int kCellThreadsFew = 64;

// One launch of a kernel template <NT, MAT, MINB, TAPE>; material: the id every
// instance of the launch uses (plasticine 5 and jelly 0 have kernels without
// the other materials' code), or -1 when they differ.
#define EMPM_CELL_LAUNCH(kernel, min_ctas, tape, n, few, material, stream, ...)                                        \
    do {                                                                                                             \
        const int nt_ = (few) ? kCellThreadsFew : kCellThreads;                                                      \
        const int g_ = ((n) + nt_ - 1) / nt_;                                                                        \
        if (few) {                                                                                                   \
            if ((material) == 5) kernel<kCellThreadsFew, 5, 1, tape><<<g_, nt_, 0, stream>>>(__VA_ARGS__);                 \
            else if ((material) == 0) kernel<kCellThreadsFew, 0, 1, tape><<<g_, nt_, 0, stream>>>(__VA_ARGS__);            \
            else kernel<kCellThreadsFew, -1, 1, tape><<<g_, nt_, 0, stream>>>(__VA_ARGS__);                                \
        } else {                                                                                                     \
            if ((material) == 5) kernel<kCellThreads, 5, min_ctas, tape><<<g_, nt_, 0, stream>>>(__VA_ARGS__);             \
            else if ((material) == 0) kernel<kCellThreads, 0, min_ctas, tape><<<g_, nt_, 0, stream>>>(__VA_ARGS__);        \
            else kernel<kCellThreads, -1, min_ctas, tape><<<g_, nt_, 0, stream>>>(__VA_ARGS__);                            \
        }                                                                                                            \
    } while (0)

static inline void launch_g2p2g_store(bool few, cudaStream_t s, const MaterialArrays& M, const Launch& L,
                                      int g2p_table, const float4* vel, float4* mom, unsigned char* flags,
                                      const SegmentStoreArgs& a, int material) {
    EMPM_CELL_LAUNCH(k_g2p2g_store, EMPM_FUSED_MIN_CTAS, true, L.n_total, few, material, s, M, L, g2p_table, vel, mom, flags, a);
}

template <bool TAPE>
static inline void launch_g2p2g(bool few, cudaStream_t s, const ParticleArrays& P, const MaterialArrays& M,
                                const F9Planes& Fe, const Launch& L, int g2p_table, const float4* vel, float4* mom,
                                unsigned char* flags, int material) {
    EMPM_CELL_LAUNCH(k_g2p2g, EMPM_FUSED_MIN_CTAS, TAPE, L.n_total, few, material, s, P, M, Fe, L, g2p_table, vel, mom, flags);
}

template <bool TAPE>
static inline void launch_p2g_cells(bool few, cudaStream_t s, const ParticleArrays& P, const MaterialArrays& M,
                                    const F9Planes& Fe, const Launch& L, float4* mom, unsigned char* flags,
                                    int material, const int* order = nullptr) {
    EMPM_CELL_LAUNCH(k_p2g_cells, EMPM_P2G_MIN_CTAS, TAPE, L.n_total, few, material, s, P, M, Fe, L, mom, flags, order);
}

// -------------------------------------------------------------------------
// sorted path, optional: shared-memory node tiles over chunks of particles
// -------------------------------------------------------------------------
constexpr int TILE_THREADS = 256;     // = chunk size

struct ChunkList {
    const int2* chunks;    // (first sorted index, count); never spans two 4^3 blocks
    const int*  nchunks;   // device count
};

__device__ __forceinline__ float sel3(const float (&a)[3], int i) { return i == 0 ? a[0] : (i == 1 ? a[1] : a[2]); }

// one node contribution with runtime stencil offsets (no local-memory indexing)
__device__ __forceinline__ float4 p2g_node_dyn(const P2GPre& p, int i, int j, int k) {
    const Stencil& st = p.st;
    const float wx = sel3(st.w[0], i), wy = sel3(st.w[1], j), wz = sel3(st.w[2], k);
    const float dwx = sel3(st.dw[0], i), dwy = sel3(st.dw[1], j), dwz = sel3(st.dw[2], k);
    const V3 a = p.a + (float)i * col(p.B, 0) + (float)j * col(p.B, 1) + (float)k * col(p.B, 2);
    const float wm = (wx * wy * wz) * p.m;
    const V3 c = wm * a + (dwx * wy * wz) * col(p.S, 0) + (wx * dwy * wz) * col(p.S, 1) + (wx * wy * dwz) * col(p.S, 2);
    return make_float4(c.x, c.y, c.z, wm);
}

struct TileBox {
    int o[3];   // origin node
    int e[3];   // extent in nodes
    int count;  // e0 * e1 * e2
};

// bounding box of the chunk's stencils (base .. base + 2) in shared memory
__device__ __forceinline__ TileBox chunk_box(bool active, const int (&b)[3], int* s_min, int* s_max) {
    if (threadIdx.x < 3) { s_min[threadIdx.x] = INT_MAX; s_max[threadIdx.x] = INT_MIN; }
    __syncthreads();
    int mn[3], mx[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) { mn[a] = active ? b[a] : INT_MAX; mx[a] = active ? b[a] : INT_MIN; }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1)
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            mn[a] = min(mn[a], __shfl_xor_sync(0xffffffffu, mn[a], d));
            mx[a] = max(mx[a], __shfl_xor_sync(0xffffffffu, mx[a], d));
        }
    if ((threadIdx.x & 31) == 0)
#pragma unroll
        for (int a = 0; a < 3; ++a) { atomicMin(s_min + a, mn[a]); atomicMax(s_max + a, mx[a]); }
    __syncthreads();
    TileBox tb;
    tb.count = 1;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        tb.o[a] = s_min[a];
        tb.e[a] = s_max[a] - s_min[a] + 3;
        tb.count *= tb.e[a];
    }
    if (s_min[0] == INT_MAX) tb.count = 0;
    return tb;
}

struct TiledArgs {
    ParticleArrays P;
    MaterialArrays M;
    F9Planes Fe;
    Launch L;
    ChunkList cl;
    float4* grid;             // P2G: accumulation; G2P: node velocities
    unsigned char* flags;     // P2G marks touched blocks
    ParticleArrays out;       // G2P output
    int tile_cap;             // nodes in the shared tile
};

__global__ void __launch_bounds__(TILE_THREADS, 2) k_p2g_tiled(const TiledArgs a) {
    extern __shared__ float4 tile[];
    __shared__ int s_min[3], s_max[3];
    const int nch = *a.cl.nchunks;
    for (int ci = blockIdx.x; ci < nch; ci += gridDim.x) {
        const int2 ch = a.cl.chunks[ci];
        const StepConsts c = consts_of(a.L, find_instance_particle(a.L, ch.x));
        const float dt = c.step->dt;
        const int p = ch.x + (int)threadIdx.x;
        bool active = threadIdx.x < (unsigned)ch.y;
        int base[3] = {0, 0, 0};
        if (active) {
            const float4 xm = __ldg(a.P.x + p);
            base[0] = base_node(xm.x, c.inv_dx);
            base[1] = base_node(xm.y, c.inv_dx);
            base[2] = base_node(xm.z, c.inv_dx);
            if (a.M.sel && __ldg(a.M.sel + p) != 0) active = false;
        }
        const TileBox tb = chunk_box(active, base, s_min, s_max);
        const bool use_tile = tb.count > 0 && tb.count <= a.tile_cap;
        if (use_tile)
            for (int t = threadIdx.x; t < tb.count; t += TILE_THREADS) tile[t] = make_float4(0.f, 0.f, 0.f, 0.f);
        __syncthreads();
        if (active) {
            P2GParticle q;
            if (prepare_particle(a.P, a.M, a.Fe, c, p, q)) {
                if (use_tile) {
                    const P2GPre pre = p2g_pre(q, c.dx, c.inv_dx, dt);
                    // stagger the 27 stencil offsets across lanes so particles of the
                    // same cell do not hit the same shared-memory node together
                    int s = (int)(threadIdx.x % 27u);
                    int i = s / 9, j = (s / 3) % 3, k = s % 3;
                    const int li0 = base_clamp(q.st.b[0]) - tb.o[0], lj0 = base_clamp(q.st.b[1]) - tb.o[1],
                              lk0 = base_clamp(q.st.b[2]) - tb.o[2];
                    for (int it = 0; it < 27; ++it) {
                        const float4 v = p2g_node_dyn(pre, i, j, k);
                        float* dst = reinterpret_cast<float*>(tile + ((li0 + i) * tb.e[1] + (lj0 + j)) * tb.e[2] + (lk0 + k));
                        atomicAdd(dst + 0, v.x);
                        atomicAdd(dst + 1, v.y);
                        atomicAdd(dst + 2, v.z);
                        atomicAdd(dst + 3, v.w);
                        if (++k == 3) { k = 0; if (++j == 3) { j = 0; if (++i == 3) i = 0; } }
                    }
                } else {
                    scatter_global(q, c, a.grid, a.flags);
                }
            }
        }
        __syncthreads();
        if (use_tile) {
            const int e12 = tb.e[1] * tb.e[2];
            for (int t = threadIdx.x; t < tb.count; t += TILE_THREADS) {
                const float4 v = tile[t];
                if (v.w == 0.f && v.x == 0.f && v.y == 0.f && v.z == 0.f) continue;
                const int gi = tb.o[0] + t / e12, gj = tb.o[1] + (t / tb.e[2]) % tb.e[1], gk = tb.o[2] + t % tb.e[2];
                if (gi < 0 || gj < 0 || gk < 0 || gi >= c.G || gj >= c.G || gk >= c.G) {
                    atomicOr(c.status, EMPM_STATUS_OUT_OF_BAND);
                    continue;
                }
                red_add_v4(a.grid + gaddr(c, gi, gj, gk), v);
            }
            // mark the 4^3 blocks the tile overlaps
            const int lo[3] = {max(tb.o[0], 0) >> 2, max(tb.o[1], 0) >> 2, max(tb.o[2], 0) >> 2};
            const int hi[3] = {min(tb.o[0] + tb.e[0] - 1, c.G - 1) >> 2, min(tb.o[1] + tb.e[1] - 1, c.G - 1) >> 2,
                               min(tb.o[2] + tb.e[2] - 1, c.G - 1) >> 2};
            const int n0 = hi[0] - lo[0] + 1, n1 = hi[1] - lo[1] + 1, n2 = hi[2] - lo[2] + 1;
            const int nmark = (n0 > 0 && n1 > 0 && n2 > 0) ? n0 * n1 * n2 : 0;
            for (int t = threadIdx.x; t < nmark; t += TILE_THREADS) {
                const int bi = lo[0] + t / (n1 * n2), bj = lo[1] + (t / n2) % n1, bk = lo[2] + t % n2;
                a.flags[c.boff + (bi * c.NB + bj) * c.NB + bk] = 1;
            }
        }
        __syncthreads();
    }
}

// Node velocities from the chunk's shared-memory tile (the stencil lies in it).
struct TileFetch {
    const float4* tile;
    int o0, o1, o2, e1, e2;
    struct Bound {
        const float4* tile;
        int x[3], y[3], z[3];   // tile index of node (i, j, k) = x[i] + y[j] + z[k]
        __device__ __forceinline__ V3 operator()(int i, int j, int k) const {
            const float4 g = tile[x[i] + y[j] + z[k]];
            return v3(g.x, g.y, g.z);
        }
    };
    __device__ __forceinline__ Bound bind(const Stencil& st, bool) const {
        Bound b;
        b.tile = tile;
#pragma unroll
        for (int o = 0; o < 3; ++o) {
            b.x[o] = (st.b[0] + o - o0) * e1 * e2;
            b.y[o] = (st.b[1] + o - o1) * e2;
            b.z[o] = st.b[2] + o - o2;
        }
        return b;
    }
};

__global__ void __launch_bounds__(TILE_THREADS, 2) k_g2p_tiled(const TiledArgs a) {
    extern __shared__ float4 tile[];
    __shared__ int s_min[3], s_max[3];
    const int nch = *a.cl.nchunks;
    for (int ci = blockIdx.x; ci < nch; ci += gridDim.x) {
        const int2 ch = a.cl.chunks[ci];
        const StepConsts c = consts_of(a.L, find_instance_particle(a.L, ch.x));
        const int p = ch.x + (int)threadIdx.x;
        const bool active = threadIdx.x < (unsigned)ch.y;
        bool stenciled = active;
        int base[3] = {0, 0, 0};
        if (active) {
            if (a.M.sel && __ldg(a.M.sel + p) != 0) stenciled = false;
            const float4 xm = __ldg(a.P.x + p);
            base[0] = base_node(xm.x, c.inv_dx);
            base[1] = base_node(xm.y, c.inv_dx);
            base[2] = base_node(xm.z, c.inv_dx);
        }
        const TileBox tb = chunk_box(stenciled, base, s_min, s_max);
        const bool use_tile = tb.count > 0 && tb.count <= a.tile_cap && tb.o[0] >= 0 && tb.o[1] >= 0 && tb.o[2] >= 0 &&
                              tb.o[0] + tb.e[0] <= c.G && tb.o[1] + tb.e[1] <= c.G && tb.o[2] + tb.e[2] <= c.G;
        if (use_tile) {
            const int e12 = tb.e[1] * tb.e[2];
            for (int t = threadIdx.x; t < tb.count; t += TILE_THREADS) {
                const int gi = tb.o[0] + t / e12, gj = tb.o[1] + (t / tb.e[2]) % tb.e[1], gk = tb.o[2] + t % tb.e[2];
                tile[t] = __ldg(a.grid + gaddr(c, gi, gj, gk));
            }
        }
        __syncthreads();
        if (active) {
            if (use_tile) {
                TileFetch f{tile, tb.o[0], tb.o[1], tb.o[2], tb.e[1], tb.e[2]};
                g2p_particle(a.P, a.Fe, a.M, a.out, c, p, f);
            } else {
                GlobalFetch f{a.grid, &c};
                g2p_particle(a.P, a.Fe, a.M, a.out, c, p, f);
            }
        }
        __syncthreads();
    }
}

}  // namespace empm
