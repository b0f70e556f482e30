// kernels_chunk.cuh -- FP32 path: the scatters over chunks of the sorted order, and the
// gathers by particle.
//
// A warp takes up to 32 consecutive particles of the cell-sorted order (a chunk).
// First one lane per particle loads its inputs, forms its stencil base and
// weights and leaves them as a record in shared memory, the particles of equal
// stencil base side by side (chunk_groups; a particle that has left its cell
// since the sort joins the group of its new cell or makes one of its own).  Then
// the groups are summed one after another: the two half-warps take alternate
// particles, and lane (i, j) of a half sums the contributions to the four nodes
// (base + (i, j, 0..3)) in registers.  At the end of a group the halves are
// added and every node gets one red.global.add.v4.f32.  So a particle's inputs
// are read and its weights formed once (warp items of 8 particles do it on 4
// lanes each), the sums over particles need no shuffles, and a cell's particles
// reach memory in one reduction per node and chunk.
//
// With w = n0 n1 n2 and d = (d0, d1, d2) a node's contribution is
//   w (b + A d) = n2 (n0n1 b + n0d0n1 A_0 + n0n1d1 A_1) + n2d2 n0n1 A_2
// (A_c: column c of A), so a lane forms the bracket once per particle and
// spends 2 multiply-adds per node and component on it.
//
// The chunk count is known on the host, so a launch is one block per 4 chunks,
// balanced by the hardware; no item list is read.
//
// Measured per step on the 64^3, 267k-particle rollout of 200 steps (sums of
// event times, which add about 3 us a launch): P2G 28.7 us against 51.6 us for
// the warp items, the adjoint scatter 40.2 against 61.6 us; on 301k particles at
// 8 per cell 36.4 / 50.7 and 42.4 / 56.7 us.  Two thirds of the L1 data pipe's
// cycles go to reading the records (25 words per lane for 2 particles), so that
// pipe bounds the sums; one particle per warp pass instead of two (8 sums per
// lane) read 21 words per particle.  Groups of strays cost: without the
// grouping (a group per run of the sorted order) 32.8 and 42.6 us.
#pragma once
#include "kernels_warp.cuh"

namespace dmpm {

// Resident blocks per SM the compiler budgets registers for: 8 of 128 threads
// (64 registers, no spills), 180 KB of records per SM
#ifndef DMPM_CHUNK_THREADS
#define DMPM_CHUNK_THREADS 128
#endif
#ifndef DMPM_CHUNK_P2G_MINB
#define DMPM_CHUNK_P2G_MINB 8
#endif
#ifndef DMPM_CHUNK_SCATTER_MINB
#define DMPM_CHUNK_SCATTER_MINB 8
#endif

// Shared-memory record of one particle (floats):
//   [2i], [2i+1]       n0[i], n0[i] d0[i]
//   [8+2j], [9+2j]     n1[j], n1[j] d1[j]
//   [16+4h .. 19+4h]   n2[2h], n2[2h+1], n2[2h] d2[2h], n2[2h+1] d2[2h+1]   (h = 0, 1)
//   [24 .. 27]         b (3) and the value summed into the 4th component
//   [28 .. 36]         A, column-major
// 44 floats apart, so that 8 lanes writing 16 bytes each cover all 32 banks
// and the records two half-warps read together fall into different banks.
constexpr int kRecFloats = 44;

// geometry of a chunk's lane or group
template <bool BATCH> __device__ __forceinline__ const GridGeom& chunk_geo(const WArgs& a, int inst) {
    if constexpr (BATCH) return a.ig[inst].g;
    else return a.geo;
}

__device__ __forceinline__ void chunk_record(float* rec, const float t[3], float dx, const float b[4], const m3<float>& A) {
    float4* r4 = reinterpret_cast<float4*>(rec);
    float n[4], e[4];
#pragma unroll
    for (int c = 0; c < 3; c++) {
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const float q = (float)k - t[c];
            n[k] = bsp(q);
            e[k] = n[k] * (q * dx);
        }
        if (c < 2) {
            r4[2 * c] = make_float4(n[0], e[0], n[1], e[1]);
            r4[2 * c + 1] = make_float4(n[2], e[2], n[3], e[3]);
        } else {
            r4[4] = make_float4(n[0], n[1], e[0], e[1]);
            r4[5] = make_float4(n[2], n[3], e[2], e[3]);
        }
    }
    r4[6] = make_float4(b[0], b[1], b[2], b[3]);
    r4[7] = make_float4(A.a[0][0], A.a[1][0], A.a[2][0], A.a[0][1]);
    r4[8] = make_float4(A.a[1][1], A.a[2][1], A.a[0][2], A.a[1][2]);
    rec[36] = A.a[2][2];
}

// The chunk's groups of equal stencil bases: a lane's record slot (the groups
// one after another, in the order of their first lanes), and for the first lane
// of a group its first slot and size.  Every lane of the warp calls it.
struct ChunkGroups {
    int slot, first, size;
    unsigned leaders;  // the groups' first lanes
};
template <bool GENERAL> __device__ __forceinline__ ChunkGroups chunk_groups(uint32_t key, bool valid) {
    const int lane = threadIdx.x & 31;
    const unsigned vm = __ballot_sync(0xffffffffu, valid);
    const unsigned m = GENERAL ? (vm & (1u << lane)) : (__match_any_sync(0xffffffffu, key) & vm);
    ChunkGroups g;
    const bool lead = valid && (m & ((1u << lane) - 1u)) == 0u;
    g.size = __popc(m);
    int x = lead ? g.size : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    g.first = x - (lead ? g.size : 0);
    g.slot = __shfl_sync(0xffffffffu, g.first, m ? __ffs(m) - 1 : 0) + __popc(m & ((1u << lane) - 1u));
    g.leaders = __ballot_sync(0xffffffffu, lead);
    return g;
}

// Sum the chunk's records group by group into dst.  NC: components (4: the 4th
// is w b[3]; 3: the 4th is left alone).  Every lane of the warp calls it.
template <bool BATCH, int NC>
__device__ __forceinline__ void chunk_scatter(const WArgs& a, const float* rec, const int base[3], int inst,
                                              const ChunkGroups& grp, node4<float>* dst) {
    const int lane = threadIdx.x & 31, hf = lane >> 4, i = (lane >> 2) & 3, j = lane & 3;
    for (unsigned left = grp.leaders; left; left &= left - 1) {
        const int lead = __ffs(left) - 1;
        const int s = __shfl_sync(0xffffffffu, grp.first, lead), e = s + __shfl_sync(0xffffffffu, grp.size, lead);
        // slots 0, 1 are the nodes this half keeps (k = 2 hf, 2 hf + 1), 2, 3 those it hands over
        float acc[4][NC];
#pragma unroll
        for (int k = 0; k < 4; k++)
#pragma unroll
            for (int c = 0; c < NC; c++) acc[k][c] = 0.f;
        auto add = [&](const float* r, bool in) {
            float2 w0 = *reinterpret_cast<const float2*>(r + 2 * i);
            const float2 w1 = *reinterpret_cast<const float2*>(r + 8 + 2 * j);
            const float4 wa = *reinterpret_cast<const float4*>(r + 16 + 4 * hf);
            const float4 wb = *reinterpret_cast<const float4*>(r + 20 - 4 * hf);
            const float4 b = *reinterpret_cast<const float4*>(r + 24);
            const float4 A0 = *reinterpret_cast<const float4*>(r + 28);
            const float4 A1 = *reinterpret_cast<const float4*>(r + 32);
            const float A22 = r[36];
            if (!in) w0 = make_float2(0.f, 0.f);
            const float a0 = w0.x * w1.x, a1 = w0.y * w1.x, a2 = w0.x * w1.y;
            const float h[3] = {a0 * b.x + a1 * A0.x + a2 * A0.w, a0 * b.y + a1 * A0.y + a2 * A1.x,
                                a0 * b.z + a1 * A0.z + a2 * A1.y};
            const float g[3] = {a0 * A1.z, a0 * A1.w, a0 * A22};
            const float n2[4] = {wa.x, wa.y, wb.x, wb.y}, e2[4] = {wa.z, wa.w, wb.z, wb.w};
            const float am = a0 * b.w;
#pragma unroll
            for (int k = 0; k < 4; k++) {
#pragma unroll
                for (int c = 0; c < 3; c++) acc[k][c] = fmaf(e2[k], g[c], fmaf(n2[k], h[c], acc[k][c]));
                if (NC == 4) acc[k][3] += n2[k] * am;
            }
        };
        const float* r = rec + (s + hf) * kRecFloats;
#pragma unroll 2
        for (int m = (e - s) >> 1; m > 0; m--, r += 2 * kRecFloats) add(r, true);
        // an odd group's last particle: the second half-warp adds nothing
        if ((e - s) & 1) add(rec + (e - 1) * kRecFloats, hf == 0);
#pragma unroll
        for (int k = 0; k < 2; k++)
#pragma unroll
            for (int c = 0; c < NC; c++) acc[k][c] += __shfl_xor_sync(0xffffffffu, acc[k + 2][c], 16);
        const int b0 = __shfl_sync(0xffffffffu, base[0], lead), b1 = __shfl_sync(0xffffffffu, base[1], lead),
                  b2 = __shfl_sync(0xffffffffu, base[2], lead);
        const int in_ = BATCH ? __shfl_sync(0xffffffffu, inst, lead) : 0;
        const GridGeom& g = chunk_geo<BATCH>(a, in_);
        const int gi = b0 + i, gj = b1 + j, gk = b2 + 2 * hf;
        if ((unsigned)gi < (unsigned)g.dim[0] && (unsigned)gj < (unsigned)g.dim[1]) {
            int node = (gi * g.dim[1] + gj) * g.dim[2] + gk;
            if (BATCH) node += a.ig[in_].goff;
#pragma unroll
            for (int k = 0; k < 2; k++) {
                const float m = NC == 4 ? acc[k][NC - 1] : 0.f;
                if ((unsigned)(gk + k) < (unsigned)g.dim[2] &&
                    (acc[k][0] != 0.f || acc[k][1] != 0.f || acc[k][2] != 0.f || m != 0.f))
                    red_add4(dst + node + k, acc[k][0], acc[k][1], acc[k][2], m);
            }
        }
    }
}

// the cell key of a lane's particle now (the sort's keys are those of an earlier step)
template <bool BATCH> __device__ __forceinline__ uint32_t chunk_key(const WArgs& a, int inst, const int base[3]) {
    const uint32_t k = cell_key(base, chunk_geo<BATCH>(a, inst).dim);
    return BATCH ? a.ig[inst].koff + k : k;
}

// The chunk's particle of this lane: its index (the first of the chunk for
// lanes past the end), instance, and the chunk's particle count.
struct ChunkLane {
    int p, inst, cnt;
    bool valid;
};
template <bool BATCH> __device__ __forceinline__ ChunkLane chunk_lane(const WArgs& a) {
    ChunkLane L;
    const int lane = threadIdx.x & 31, q0 = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * a.chunk;
    L.cnt = min(a.chunk, a.n - q0);  // <= 0: the warp has no particles
    L.valid = lane < L.cnt;
    L.p = L.cnt > 0 ? (int)a.items.order[q0 + (L.valid ? lane : 0)] : 0;
    L.inst = BATCH ? (int)a.pinst[L.p] : 0;
    return L;
}

// P2G: m_g += w m_p;  p_g += w (m_p v (1 - dt drag) + G (x_g - x_p))
template <bool BATCH, bool GENERAL>
__global__ void __launch_bounds__(DMPM_CHUNK_THREADS, DMPM_CHUNK_P2G_MINB) k_p2g_c(WArgs a) {
    __shared__ __align__(16) float s_rec[DMPM_CHUNK_THREADS * kRecFloats];
    const ChunkLane L = chunk_lane<BATCH>(a);
    if (L.cnt <= 0) return;
    const int have = !BATCH && a.box && (threadIdx.x & 31) < 6 ? *(volatile int*)(a.box + (threadIdx.x & 31)) : 0;
    float* rec = s_rec + (threadIdx.x & ~31) * kRecFloats;
    float t[3];
    int base[3];
    load_x_base(a.st, a.npl, L.p, chunk_geo<BATCH>(a, L.inst), t, base, a.xlo);
    const ChunkGroups grp = chunk_groups<GENERAL>(chunk_key<BATCH>(a, L.inst, base), L.valid);
    if (!BATCH && a.box) widen_box(a.box, have, a.geo, base, L.valid);
    {
        const float mp = a.cst[(size_t)KM * a.np + L.p], damp = 1.f - a.dt * a.drag;
        float b[4];
#pragma unroll
        for (int c = 0; c < 3; c++) b[c] = mp * a.st[(size_t)(PV + c) * a.npl + L.p] * damp;
        b[3] = mp;
        const m3<float> G = load_m3((const float*)a.G, a.npl, L.p);
        if (L.valid) chunk_record(rec + grp.slot * kRecFloats, t, (float)a.geo.dx, b, G);
    }
    __syncwarp();
    chunk_scatter<BATCH, 4>(a, rec, base, L.inst, grp, a.grid);
}

// adjoint G2P scatter: dLdv_g += w (dLdv_next + 3/dx^2 dLdC_next (x_g - x_p))
// (BackPropagation.cpp:14-44), the sources (adj_sources) left in adjn for the gather
template <bool EXACT, bool BATCH, bool GENERAL>
__global__ void __launch_bounds__(DMPM_CHUNK_THREADS, DMPM_CHUNK_SCATTER_MINB) k_adj_scatter_c(WArgs a) {
    __shared__ __align__(16) float s_rec[DMPM_CHUNK_THREADS * kRecFloats];
    const ChunkLane L = chunk_lane<BATCH>(a);
    if (L.cnt <= 0) return;
    float* rec = s_rec + (threadIdx.x & ~31) * kRecFloats;
    float t[3];
    int base[3];
    load_x_base(a.st, a.npl, L.p, chunk_geo<BATCH>(a, L.inst), t, base, a.xlo);
    const ChunkGroups grp = chunk_groups<GENERAL>(chunk_key<BATCH>(a, L.inst, base), L.valid);
    {
        const size_t np = a.np;
        float b[4];
        m3<float> Cn;
        adj_sources<EXACT>(a, L.p, b, Cn);
        b[3] = 0.f;
        if (L.valid) {
#pragma unroll
            for (int c = 0; c < 3; c++) a.adjn[(size_t)c * np + L.p] = b[c];
            store_m3(a.adjn + 3 * np, np, L.p, Cn);
            if (a.dbg_vnext) {
#pragma unroll
                for (int c = 0; c < 3; c++) a.dbg_vnext[(size_t)c * np + L.p] = b[c];
            }
            if (a.dbg_Cnext) store_m3(a.dbg_Cnext, np, L.p, Cn);
            const float dx = (float)a.geo.dx;
            chunk_record(rec + grp.slot * kRecFloats, t, dx, b, (3.f / (dx * dx)) * Cn);
        }
    }
    __syncwarp();
    chunk_scatter<BATCH, 3>(a, rec, base, L.inst, grp, a.gadj);
}

// Particles per warp: 32 gives the fewest reductions and record reads per
// particle, fewer spread a small cloud over the SMs.  P2G / adjoint scatter us
// at 8, 16, 32 per warp: 8.7k particles 9.9 / 10.1 / 11.7 and 10.3 / 10.5 /
// 12.3; 19k 11.1 / 10.6 / 12.4 and 11.8 / 11.8 / 12.6; 33k 13.3 / 12.7 / 12.6 and
// 14.8 / 14.1 / 13.1; 79k 20.5 / 17.2 / 16.6 and 24.4 / 20.9 / 18.6; 267k 43.9 /
// 32.5 / 29.0 and 58.3 / 43.4 / 39.8.  So: the most that leave 8 warps for each of
// 148 SMs.
inline int scatter_chunk(int n) {
    const int warps = 148 * 8;
    return n >= 32 * warps ? 32 : n >= 16 * warps ? 16 : 8;
}
// The FP64 path's, whose node adds are four atomics each: fewer of them sooner pay
// for idle SMs.  P2G and adjoint scatter together: 3.0k particles 27.8 / 30.3 / 36.9,
// 6.3k 30.9 / 29.7 / 33.3, 13k 44.9 / 40.6 / 36.7, 19k 52.6 / 42.2 / 43.8, 33k 71.4 /
// 57.1 / 52.8, 70k 110.8 / 82.6 / 72.7.
inline int scatter_chunk64(int n) {
    const int warps = 148 * 5 / 2;
    return n >= 32 * warps ? 32 : n >= 16 * warps ? 16 : 8;
}
// blocks of a chunk kernel over n particles, chunk particles a warp
inline unsigned chunk_blocks(int n, int chunk) {
    const int per = chunk * (DMPM_CHUNK_THREADS / 32);
    return (unsigned)((n + per - 1) / per);
}

// Per-axis stencil offsets d = x_g - x, weights N(d / dx) and slopes of the
// four nodes k = 0..3 of the stencil, from the lattice coordinate t of the
// particle (load_x_base): d = (k - t) dx.
__device__ __forceinline__ void axis_stencil(float t, float dx, float n[4], float d[4], float* s) {
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const float q = (float)k - t;
        d[k] = q * dx;
        n[k] = bsp(q);
        if (s) s[k] = bsp_slope(q);
    }
}

// ------------------------------------------------------------------ adjoint gather + finalize
// One thread per particle, reading the nodes where they lie.  Particles are taken as
// they are stored, not in cell order: their 110 planes then come in whole sectors,
// and the nodes of a cloud lie in L2 whichever particle asks.  In a spatial order
// (lattice, cell order) a warp's reads are broadcasts from L1 or nearly so; in a
// random one the planes would cost a sector per value in cell order.  Gather and
// G2P at 267k particles in lattice order 92.4 and 47.4 us (in cell order 99.1 and
// 49.9), in random order 126.5 and 66.3 (289.9 and 157.2); 2.0M in lattice order 440
// and 244 (471 and 275); stored in cell order the same.  The thread keeps the 18 sums of its particle in registers
// and goes on to the finalize with them (as two kernels the sums made a round
// trip of 144 bytes per particle, and the finalize a second and a third launch).
// Small clouds give a particle four threads, one per stencil slab (SPLIT).
//
// Measured per step on the 64^3, 267k-particle rollout (event times, in cell order as
// are the rest): 98 us, and the warp-item gather with the two finalize kernels behind
// it 82.6 + 41.4 (+ 14.6 beside them); 79k particles with the reference's adjoint 33
// against 27 + 57 us; 8.7k particles 14.7 against 12.6 + 8.7.  The node sums take
// 55 us of the 98 (in a kernel of their own): 22.3 M warp instructions at 42 % issue with 16 warps per
// SM, which wait for L1 and L2 at each of the 16 stencil rows.  What did not help:
// the warp's nodes copied to shared memory as one box first (58.6 us: the waits
// went, 8 M instructions came), 12 warps without spills or 20 with more (58 /
// 71-80 us), all of the finalize's inputs staged or prefetched during the sums
// (within 2 us either way).

// copy 4 bytes to shared memory asynchronously, through L1
__device__ __forceinline__ void async4(float* dst, const float* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}
__device__ __forceinline__ void async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// Two floats in one 64-bit register pair: sm_100a multiplies and adds both in one
// instruction.
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pk(float a, float b) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void unpk(f32x2 p, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(p)); }
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ float sum2(f32x2 p) {
    float a, b;
    unpk(p, a, b);
    return a + b;
}
// the record pair (dLdp, dLdm), (v, m) of a node: one 32-byte load
__device__ __forceinline__ void load_pair(const node4<float>* p, f32x2 (&f)[4]) {
    asm("ld.global.nc.v4.b64 {%0, %1, %2, %3}, [%4];" : "=l"(f[0]), "=l"(f[1]), "=l"(f[2]), "=l"(f[3]) : "l"(p));
}
// Nodes of a particle's stencil by offset (i, j, k) from its base.  INSIDE: the
// whole stencil lies in the grid; otherwise nodes outside it read as zero.  A grid
// has up to 2e9 nodes, so a stencil inside it spans less than 2^31 single records and
// 2^32 of pairs; one that reaches over the grid's edge may be longer than the grid,
// and its rows need 64 bits.  At 267k particles, in cell order, G2P 49.6 us and the
// gather 99.0 (49.5 and 98.6 in ints throughout; with unsigned offsets in G2P too
// 50.3, with 64 bits for all stencils the gather 99.8).
template <bool INSIDE, int R> struct StencilNodes {
    const node4<float>* g;  // the base node's first record (dereferenced inside the grid only)
    unsigned si, sj;        // records per slab and row
    int b0, b1, b2, d0, d1, d2;
    DMPM_HD StencilNodes(const node4<float>* grid, const GridGeom& geo, int goff, const int base[3])
        : g(grid + R * (((ptrdiff_t)base[0] * geo.dim[1] + base[1]) * geo.dim[2] + base[2] + goff)),
          si((unsigned)R * (unsigned)(geo.dim[1] * geo.dim[2])), sj((unsigned)R * (unsigned)geo.dim[2]), b0(base[0]),
          b1(base[1]), b2(base[2]), d0(geo.dim[0]), d1(geo.dim[1]), d2(geo.dim[2]) {}
    DMPM_HD const node4<float>* row(int i, int j) const {
        if (INSIDE && R == 1) return g + (i * (int)si + j * (int)sj);
        return g + (INSIDE ? (size_t)((unsigned)i * si + (unsigned)j * sj) : (size_t)i * si + (size_t)j * sj);
    }
    DMPM_HD bool in(int i, int j, int k) const {
        return INSIDE || ((unsigned)(b0 + i) < (unsigned)d0 && (unsigned)(b1 + j) < (unsigned)d1 &&
                          (unsigned)(b2 + k) < (unsigned)d2);
    }
};
__device__ __forceinline__ bool stencil_inside(const GridGeom& g, const int base[3]) {
    bool in = true;
#pragma unroll
    for (int c = 0; c < 3; c++) in &= base[c] >= 0 && base[c] + 3 < g.dim[c];
    return in;
}

// a node's (v.x, v.y), (v.z, m): one 16-byte load
__device__ __forceinline__ void load_node(const node4<float>* p, f32x2 (&f)[2]) {
    asm("ld.global.nc.v2.b64 {%0, %1}, [%2];" : "=l"(f[0]), "=l"(f[1]) : "l"(p));
}
// Start reading the stencils of the warp's first and last particle into L1, R
// records of 16 bytes per node: copies to a word that nobody reads.
template <int R>
__device__ __forceinline__ void warm_stencils(const node4<float>* nodes, const GridGeom& g, int goff, const int base[3],
                                              float* dump) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int h = 0; h < 2; h++) {
        int o[3];
#pragma unroll
        for (int c = 0; c < 3; c++) o[c] = __shfl_sync(0xffffffffu, base[c], h ? 31 : 0);
#pragma unroll
        for (int m = 0; m < 2; m++) {
            const int gi = o[0] + 2 * m + (lane >> 4), gj = o[1] + ((lane >> 2) & 3), gk = o[2] + (lane & 3);
            if (in_grid(g, gi, gj, gk)) async4(dump, &nodes[R * (node_id(g, gi, gj, gk) + goff)].x);
        }
    }
}

// ------------------------------------------------------------------ G2P + P_op_2 (+ next stress stage)
// v' = sum w v_g;  C' = 3/dx^2 sum w v_g d^T, factored per row and slab (s: V, then
// the columns of C' / (3/dx^2), each (x, y), (z, unused)).
template <int SPLIT, class Nodes>
__device__ __forceinline__ void g2p_sums(const Nodes& f, const float t[3], float dx, f32x2 (&s)[8]) {
    float n1[4], d1[4], n2[4], d2[4];
    axis_stencil(t[1], dx, n1, d1, nullptr);
    axis_stencil(t[2], dx, n2, d2, nullptr);
#pragma unroll
    for (int c = 0; c < 8; c++) s[c] = 0;
    const int i0 = SPLIT == 4 ? (int)(threadIdx.x & 3) : 0;
#pragma unroll 1
    for (int i = i0; i < (SPLIT == 4 ? i0 + 1 : 4); i++) {
        const float q0 = (float)i - t[0], n0 = bsp(q0), e0 = n0 * (q0 * dx);
        f32x2 V[2] = {0, 0}, C1[2] = {0, 0}, C2[2] = {0, 0};
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const node4<float>* row = f.row(i, j);
            f32x2 nd[4][2];
#pragma unroll
            for (int k = 0; k < 4; k++) {
                nd[k][0] = nd[k][1] = 0;
                if (f.in(i, j, k)) load_node(row + k, nd[k]);
            }
            f32x2 Vj[2] = {0, 0}, Wj[2] = {0, 0};
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const float e = n2[k] * d2[k];
                const f32x2 nn = pk(n2[k], n2[k]), ee = pk(e, e);
#pragma unroll
                for (int c = 0; c < 2; c++) {
                    Vj[c] = fma2(nn, nd[k][c], Vj[c]);
                    Wj[c] = fma2(ee, nd[k][c], Wj[c]);
                }
            }
            const float e1 = n1[j] * d1[j];
            const f32x2 nn = pk(n1[j], n1[j]), ee = pk(e1, e1);
#pragma unroll
            for (int c = 0; c < 2; c++) {
                V[c] = fma2(nn, Vj[c], V[c]);
                C1[c] = fma2(ee, Vj[c], C1[c]);
                C2[c] = fma2(nn, Wj[c], C2[c]);
            }
        }
        const f32x2 nn = pk(n0, n0), ee = pk(e0, e0);
#pragma unroll
        for (int c = 0; c < 2; c++) {
            s[c] = fma2(nn, V[c], s[c]);
            s[2 + c] = fma2(ee, V[c], s[2 + c]);
            s[4 + c] = fma2(nn, C1[c], s[4 + c]);
            s[6 + c] = fma2(nn, C2[c], s[6 + c]);
        }
    }
}

// One thread per particle (four of small clouds) in storage order, as the adjoint
// gather.  Per step, with the next stress stage (event times; before: a CTA per
// brick octant that staged its node tile behind two barriers, 2.1 waves of them):
// 267k particles 47 against 64 us, 301k at 8 per cell 46 against 87, 2.0M 244 against
// 490, 8.7k 12.4 against 14; 3 or 5 blocks per SM each 2 us more on the first.  F' = (1 - s)(I + dt C')(F + dFc) + s F;  x' = x + dt v'.
// STRESS: also the next step's stress stage from the strain and C just formed
// (stress_particle, the arithmetic of k_stress), into a.G_next, for the first
// a.n_next particles -- one pass over the particles fewer per step.
#ifndef DMPM_CHUNK_G2P_MINB
#define DMPM_CHUNK_G2P_MINB 4
#endif
template <bool BATCH, bool STRESS, int SPLIT>
__global__ void __launch_bounds__(DMPM_CHUNK_THREADS, STRESS ? DMPM_CHUNK_G2P_MINB : 6) k_g2p_c(WArgs a) {
    __shared__ float s_dump[DMPM_CHUNK_THREADS];
    const int q = (int)((blockIdx.x * blockDim.x + threadIdx.x) / SPLIT);
    if ((q & ~(32 / SPLIT - 1)) >= a.n) return;  // the whole warp
    if (!BATCH && blockIdx.x == 0 && a.box_next) box_join(a.box_next, a.box);
    const size_t np = a.np, npl = a.npl, npn = a.npn;
    const int p = min(q, a.n - 1);
    const int inst = BATCH ? (int)a.pinst[p] : 0;
    const GridGeom& geo = chunk_geo<BATCH>(a, inst);
    const int goff = BATCH ? a.ig[inst].goff : 0;
    float t[3];
    int base[3];
    double xd[3];
    load_x_base(a.st, npl, p, geo, t, base, a.xlo, xd);
    warm_stencils<1>(a.grid, geo, goff, base, s_dump + threadIdx.x);
    async_commit();
    const m3<float> H = load_m3(a.st + (size_t)PF * npl, npl, p);
    const m3<float> D = H + load_m3(a.dfc, np, p);
    const float dx = (float)a.geo.dx, k3 = 3.f / (dx * dx);
    float s[12];
    {
        f32x2 s2[8];
        if (__all_sync(0xffffffffu, stencil_inside(geo, base)))
            g2p_sums<SPLIT>(StencilNodes<true, 1>(a.grid, geo, goff, base), t, dx, s2);
        else
            g2p_sums<SPLIT>(StencilNodes<false, 1>(a.grid, geo, goff, base), t, dx, s2);
        float skip;
#pragma unroll
        for (int c = 0; c < 4; c++) {
            unpk(s2[2 * c], s[3 * c], s[3 * c + 1]);
            unpk(s2[2 * c + 1], s[3 * c + 2], skip);
        }
    }
    if (SPLIT == 4) reduce_slabs<12>(s);
    async_wait<0>();
    if (q >= a.n || (SPLIT == 4 && (threadIdx.x & 3) != 0)) return;
    m3<float> Cn;
#pragma unroll
    for (int r = 0; r < 3; r++)
#pragma unroll
        for (int c = 0; c < 3; c++) Cn.a[r][c] = k3 * s[3 + 3 * c + r];
    bool finite = true;
#pragma unroll
    for (int c = 0; c < 3; c++) {
        const float xn = store_x(a.st_next, npn, p, c, xd[c], a.dt, s[c], a.xlo);
        a.st_next[(size_t)(PV + c) * npn + p] = s[c];
        finite &= isfinite(xn);
    }
    store_m3(a.st_next + (size_t)PC * npn, npn, p, Cn);
    // strain update H' = (1 - s)(D + dt C' (I + D)) + s H,  D = H + dFc
    m3<float> Hn;
#pragma unroll
    for (int c = 0; c < 3; c++)
#pragma unroll
        for (int r = 0; r < 3; r++) {
            const float u = D.a[r][c] + a.dt * (Cn.a[r][c] + (Cn.a[r][0] * D.a[0][c] + Cn.a[r][1] * D.a[1][c] +
                                                               Cn.a[r][2] * D.a[2][c]));
            const float hn = (1.f - a.s) * u + a.s * H.a[r][c];
            a.st_next[(size_t)(PF + r + 3 * c) * npn + p] = hn;
            Hn.a[r][c] = hn;
            finite &= isfinite(hn);
        }
    if (!finite) atomicOr(a.status, ST_NONFINITE_FWD);
    if (STRESS && p < a.n_next)
        stress_particle(a, p, Hn, load_m3(a.dfc_next, np, p), [&]() { return Cn; }, a.G_next, npn, a.P_next);
}

// The gather's sums (the algebra of kernels.cuh:k_adj_gather): g = M (9, row-major), X, u, z.
// The columns of G and of dLdC_next are read from the particle's staged inputs
// (col: 18 values, 32 floats apart) where they are needed, so that
// they hold no registers; k3 = 3/dx^2 scales the second.
template <int SPLIT, class Nodes>
__device__ __forceinline__ void gather_sums(const Nodes& f, const float t[3], float dx, float k3, float mp,
                                            const float mvp[3], const float vn[3], const float* col, float2* w1s,
                                            float (&g)[18]) {
    auto G = [&](int r, int c) { return col[(r + 3 * c) * 32]; };
    auto C = [&](int r, int c) { return col[(9 + r + 3 * c) * 32]; };
    float n2[4], d2[4], s2[4];
    axis_stencil(t[2], dx, n2, d2, s2);
#pragma unroll
    for (int j = 0; j < 4; j++) {
        const float q1 = (float)j - t[1];
        w1s[j * 32] = make_float2(bsp(q1), bsp_slope(q1));
    }
    // a node's packed fields: (o.x, o.y), (o.z, o.w), (v.x, v.y), (v.z, m); sigma is their product with
    // (h.x, h.y), (h.z, m_p), (e.x, e.y), (e.z, 0)
    const f32x2 K[4] = {pk(G(0, 2), G(1, 2)), pk(G(2, 2), 0.f), pk(k3 * C(0, 2), k3 * C(1, 2)), pk(k3 * C(2, 2), 0.f)};
    f32x2 u[2] = {0, 0}, z[2] = {0, 0}, M[3][2] = {{0, 0}, {0, 0}, {0, 0}};
    float X[3] = {0.f, 0.f, 0.f};
    const int i0 = SPLIT == 4 ? (int)(threadIdx.x & 3) : 0;
#pragma unroll 1
    for (int i = i0; i < (SPLIT == 4 ? i0 + 1 : 4); i++) {
        const float q0 = (float)i - t[0], d0 = q0 * dx, n0 = bsp(q0), s0 = bsp_slope(q0), kd0 = k3 * d0;
        const f32x2 h0[4] = {pk(mvp[0] + G(0, 0) * d0, mvp[1] + G(1, 0) * d0), pk(mvp[2] + G(2, 0) * d0, mp),
                             pk(vn[0] + C(0, 0) * kd0, vn[1] + C(1, 0) * kd0), pk(vn[2] + C(2, 0) * kd0, 0.f)};
#pragma unroll 2
        for (int j = 0; j < 4; j++) {
            const float2 ns1 = w1s[j * 32];
            const float d1 = ((float)j - t[1]) * dx, n1 = ns1.x, s1 = ns1.y, kd1 = k3 * d1;
            const node4<float>* row = f.row(i, j);
            f32x2 nd[4][4];
#pragma unroll
            for (int k = 0; k < 4; k++) {
#pragma unroll
                for (int c = 0; c < 4; c++) nd[k][c] = 0;
                if (f.in(i, j, k)) load_pair(row + 2 * k, nd[k]);
            }
            const f32x2 dd = pk(d1, d1), kd = pk(kd1, kd1);
            const f32x2 h[4] = {fma2(pk(G(0, 1), G(1, 1)), dd, h0[0]), fma2(pk(G(2, 1), 0.f), dd, h0[1]),
                                fma2(pk(C(0, 1), C(1, 1)), kd, h0[2]), fma2(pk(C(2, 1), 0.f), kd, h0[3])};
            f32x2 S = 0, T = 0, R[4] = {0, 0, 0, 0}, D[2] = {0, 0};
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const f32x2 d = pk(d2[k], d2[k]), n = pk(n2[k], n2[k]), s = pk(s2[k], s2[k]);
                const f32x2 e = mul2(n, d);
                f32x2 sig = mul2(nd[k][0], fma2(K[0], d, h[0]));
#pragma unroll
                for (int c = 1; c < 4; c++) sig = fma2(nd[k][c], fma2(K[c], d, h[c]), sig);
                S = fma2(n, sig, S);
                T = fma2(s, sig, T);
#pragma unroll
                for (int c = 0; c < 4; c++) R[c] = fma2(n, nd[k][c], R[c]);
                D[0] = fma2(e, nd[k][0], D[0]);
                D[1] = fma2(e, nd[k][1], D[1]);
            }
            const float w01 = n0 * n1, w0 = w01 * d0, w1 = w01 * d1, Sr = sum2(S), Tr = sum2(T);
            const f32x2 w = pk(w01, w01), a0 = pk(w0, w0), a1 = pk(w1, w1);
#pragma unroll
            for (int c = 0; c < 2; c++) {
                u[c] = fma2(w, R[c], u[c]);
                z[c] = fma2(w, R[2 + c], z[c]);
                M[0][c] = fma2(a0, R[c], M[0][c]);
                M[1][c] = fma2(a1, R[c], M[1][c]);
                M[2][c] = fma2(w, D[c], M[2][c]);
            }
            X[0] += (s0 * n1) * Sr;
            X[1] += (n0 * s1) * Sr;
            X[2] += w01 * Tr;
        }
    }
    float skip;
#pragma unroll
    for (int r = 0; r < 3; r++) {
        unpk(M[r][0], g[3 * r], g[3 * r + 1]);
        unpk(M[r][1], g[3 * r + 2], skip);
        g[9 + r] = X[r];
    }
    unpk(u[0], g[12], g[13]);
    unpk(u[1], g[14], skip);
    unpk(z[0], g[15], g[16]);
    unpk(z[1], g[17], skip);
    if (SPLIT == 4) reduce_slabs<18>(g);
}

// place of a staged slot in the thread's column: G (9), dLdC_next (9)
constexpr int kStaged = 18;
__host__ __device__ constexpr bool is_staged(int s) { return (s >= FS_AUX && s < FS_AUX + 9) || (s >= FS_CN && s < FS_CN + 9); }
__host__ __device__ constexpr int staged_slot(int s) { return s < FS_CN ? s - FS_AUX : 9 + s - FS_CN; }
// stage slots [lo, hi) of the finalize's inputs (fin_plane) of particle p
template <int LO, int HI> __device__ __forceinline__ void stage_slots(const WArgs& a, int p, float* col) {
#pragma unroll
    for (int s = LO; s < HI; s++) {
        size_t ld;
        const float* src = fin_plane(a, s, ld);
        async4(col + staged_slot(s) * 32, src + p);
    }
}

// the finalize's inputs: the gather's sums in registers, G and dLdC_next staged, the rest in memory
struct FinStaged {
    const WArgs* a;
    int p;
    const float* g;
    const float* col;
    __device__ __forceinline__ float operator()(int slot) const {
        if (slot < FS_F) return g[slot];
        if (is_staged(slot)) return col[staged_slot(slot) * 32];
        size_t ld;
        return fin_plane(*a, slot, ld)[p];
    }
    __device__ __forceinline__ double acc(int i) const { return a->ctrl_acc[(size_t)i * a->np + p]; }
};

// resident blocks per SM the compiler budgets registers for (128 registers)
#ifndef DMPM_CHUNK_GATHER_MINB
#define DMPM_CHUNK_GATHER_MINB 4
#endif
template <bool EXACT, bool BATCH, int SPLIT>
__global__ void __launch_bounds__(DMPM_CHUNK_THREADS, DMPM_CHUNK_GATHER_MINB) k_adj_gather_c(WArgs a) {
    __shared__ float s_col[DMPM_CHUNK_THREADS * kStaged];
    __shared__ float2 s_w1[DMPM_CHUNK_THREADS * 4];
    __shared__ float s_dump[DMPM_CHUNK_THREADS];
    const int q = (int)((blockIdx.x * blockDim.x + threadIdx.x) / SPLIT);
    if ((q & ~(32 / SPLIT - 1)) >= a.n) return;  // the whole warp
    float* col = s_col + (threadIdx.x >> 5) * 32 * kStaged + (threadIdx.x & 31);
    float2* w1s = s_w1 + (threadIdx.x >> 5) * 128 + (threadIdx.x & 31);
    const size_t np = a.np, npl = a.npl;
    const int p = min(q, a.n - 1);
    const int inst = BATCH ? (int)a.pinst[p] : 0;
    const GridGeom& geo = chunk_geo<BATCH>(a, inst);
    const int goff = BATCH ? a.ig[inst].goff : 0;
    stage_slots<FS_AUX, FS_AUX + 9>(a, p, col);
    stage_slots<FS_CN, FS_CN + 9>(a, p, col);
    float t[3];
    int base[3];
    load_x_base(a.st, npl, p, geo, t, base, a.xlo);
    warm_stencils<2>(a.gadj2, geo, goff, base, s_dump + threadIdx.x);  // 102 -> 98 us
    async_commit();
    const float dx = (float)a.geo.dx, k3 = 3.f / (dx * dx);
    const float mp = a.cst[(size_t)KM * np + p], cd = EXACT ? (1.f - a.dt * a.drag) : 1.f;
    float mvp[3], vn[3];
#pragma unroll
    for (int c = 0; c < 3; c++) {
        mvp[c] = mp * a.st[(size_t)(PV + c) * npl + p] * cd;
        vn[c] = a.adjn[(size_t)c * np + p];
    }
    async_wait<0>();
    float g[18];
    if (__all_sync(0xffffffffu, stencil_inside(geo, base)))
        gather_sums<SPLIT>(StencilNodes<true, 2>(a.gadj2, geo, goff, base), t, dx, k3, mp, mvp, vn, col, w1s, g);
    else
        gather_sums<SPLIT>(StencilNodes<false, 2>(a.gadj2, geo, goff, base), t, dx, k3, mp, mvp, vn, col, w1s, g);
    if (q < a.n && (SPLIT == 1 || (threadIdx.x & 3) == 0))
        finalize_particle<EXACT>(a, p, FinStaged{&a, p, g, col});
}

// threads per block of the one-thread-per-particle kernels: the most that leave
// two blocks for each of 148 SMs
inline int particle_threads(int n) {
    const int blocks = 148 * 2;
    return n >= 128 * blocks ? 128 : n >= 64 * blocks ? 64 : 32;
}
// Threads per particle of G2P and the gather.  Four shorten the chain of a cloud that
// leaves SMs idle and repeat the weights of each; from 19k particles they also need a
// second wave of blocks.  A step forward and back, us with four / with one: 3.0k
// particles 31.9 / 37.2, 8.7k 37.3 / 42.4, 13.1k 42.5 / 44.9, 14.4k 46.4 / 46.4, 16.0k
// 47.4 / 46.0, 19.4k 58.0 / 46.5, 26.6k 66.8 / 49.0, 39.5k 84.2 / 56.8.
inline int particle_split(int n) { return n < 14500 ? 4 : 1; }
// G2P, with the next stress stage where a.G_next is set
template <bool BATCH> inline void launch_g2p(const WArgs& a, cudaStream_t st) {
    const int split = particle_split(a.n), t = particle_threads(split * a.n);
    const unsigned b = (unsigned)((split * a.n + t - 1) / t);
    if (split == 4 && a.G_next) k_g2p_c<BATCH, true, 4><<<b, t, 0, st>>>(a);
    else if (split == 4) k_g2p_c<BATCH, false, 4><<<b, t, 0, st>>>(a);
    else if (a.G_next) k_g2p_c<BATCH, true, 1><<<b, t, 0, st>>>(a);
    else k_g2p_c<BATCH, false, 1><<<b, t, 0, st>>>(a);
}
template <bool BATCH> inline void launch_gather(const WArgs& a, bool exact, cudaStream_t st) {
    const int split = particle_split(a.n), t = particle_threads(split * a.n);
    const unsigned b = (unsigned)((split * a.n + t - 1) / t);
    if (split == 4 && exact) k_adj_gather_c<true, BATCH, 4><<<b, t, 0, st>>>(a);
    else if (split == 4) k_adj_gather_c<false, BATCH, 4><<<b, t, 0, st>>>(a);
    else if (exact) k_adj_gather_c<true, BATCH, 1><<<b, t, 0, st>>>(a);
    else k_adj_gather_c<false, BATCH, 1><<<b, t, 0, st>>>(a);
}

// ------------------------------------------------------------------ FP64 path
// P2G and the adjoint scatter of the FP64 path, as above in double.  One thread
// per particle adding each of its 64 nodes with 4 FP64 atomics took 146 and 155 us
// per step on 57.7k particles at 8 per cell; here a cell's particles reach a node
// in one round of atomics: 35 and 30 us.
// Record (doubles, 16-byte pairs): (n0, n0 d0)[4], (n1, n1 d1)[4], n2 and n2 d2 in
// pairs of nodes (2h, 2h + 1), b (4), A (9, column-major); 38 apart.
constexpr int kRec64 = 38;
__device__ __forceinline__ void chunk_record64(double* rec, const axis_w<double> (&w)[3], const double b[4],
                                               const m3<double>& A) {
    double2* r = reinterpret_cast<double2*>(rec);
#pragma unroll
    for (int c = 0; c < 2; c++)
#pragma unroll
        for (int k = 0; k < 4; k++) r[4 * c + k] = make_double2(w[c].n[k], w[c].n[k] * w[c].d[k]);
#pragma unroll
    for (int h = 0; h < 2; h++) {
        r[8 + 2 * h] = make_double2(w[2].n[2 * h], w[2].n[2 * h + 1]);
        r[9 + 2 * h] = make_double2(w[2].n[2 * h] * w[2].d[2 * h], w[2].n[2 * h + 1] * w[2].d[2 * h + 1]);
    }
    r[12] = make_double2(b[0], b[1]);
    r[13] = make_double2(b[2], b[3]);
    r[14] = make_double2(A.a[0][0], A.a[1][0]);
    r[15] = make_double2(A.a[2][0], A.a[0][1]);
    r[16] = make_double2(A.a[1][1], A.a[2][1]);
    r[17] = make_double2(A.a[0][2], A.a[1][2]);
    rec[36] = A.a[2][2];
}
template <int NC>
__device__ __forceinline__ void chunk_scatter64(const double* rec, const int base[3], const ChunkGroups& grp,
                                                const GridGeom& g, node4<double>* dst) {
    const int lane = threadIdx.x & 31, hf = lane >> 4, i = (lane >> 2) & 3, j = lane & 3;
    for (unsigned left = grp.leaders; left; left &= left - 1) {
        const int lead = __ffs(left) - 1;
        const int s = __shfl_sync(0xffffffffu, grp.first, lead), e = s + __shfl_sync(0xffffffffu, grp.size, lead);
        double acc[4][NC];
#pragma unroll
        for (int k = 0; k < 4; k++)
#pragma unroll
            for (int c = 0; c < NC; c++) acc[k][c] = 0.0;
#pragma unroll 1
        for (int q = s; q < e; q += 2) {
            const bool in = q + hf < e;
            const double* p = rec + (in ? q + hf : s) * kRec64;
            const double2* r = reinterpret_cast<const double2*>(p);
            double2 w0 = r[i];
            const double2 w1 = r[4 + j], na = r[8 + 2 * hf], ea = r[9 + 2 * hf], nb = r[10 - 2 * hf], eb = r[11 - 2 * hf];
            const double2 b01 = r[12], b23 = r[13], A0 = r[14], A1 = r[15], A2 = r[16], A3 = r[17];
            if (!in) w0 = make_double2(0.0, 0.0);
            const double a0 = w0.x * w1.x, a1 = w0.y * w1.x, a2 = w0.x * w1.y;
            const double h[3] = {a0 * b01.x + a1 * A0.x + a2 * A1.y, a0 * b01.y + a1 * A0.y + a2 * A2.x,
                                 a0 * b23.x + a1 * A1.x + a2 * A2.y};
            const double gg[3] = {a0 * A3.x, a0 * A3.y, a0 * p[36]};
            const double n2[4] = {na.x, na.y, nb.x, nb.y}, e2[4] = {ea.x, ea.y, eb.x, eb.y}, am = a0 * b23.y;
#pragma unroll
            for (int k = 0; k < 4; k++) {
#pragma unroll
                for (int c = 0; c < 3; c++) acc[k][c] += n2[k] * h[c] + e2[k] * gg[c];
                if (NC == 4) acc[k][NC - 1] += n2[k] * am;
            }
        }
#pragma unroll
        for (int k = 0; k < 2; k++)
#pragma unroll
            for (int c = 0; c < NC; c++) acc[k][c] += __shfl_xor_sync(0xffffffffu, acc[k + 2][c], 16);
        const int gi = __shfl_sync(0xffffffffu, base[0], lead) + i, gj = __shfl_sync(0xffffffffu, base[1], lead) + j,
                  gk = __shfl_sync(0xffffffffu, base[2], lead) + 2 * hf;
#pragma unroll
        for (int k = 0; k < 2; k++)
            if (in_grid(g, gi, gj, gk + k)) {
                double* n = &dst[node_id(g, gi, gj, gk + k)].x;
#pragma unroll
                for (int c = 0; c < NC; c++)
                    if (acc[k][c] != 0.0) atomicAdd(n + c, acc[k][c]);
            }
    }
}
// the lane's particle, stencil base and weights, as the FP64 path forms them
struct ChunkLane64 {
    int p, cnt, base[3];
    bool valid;
    axis_w<double> w[3];
    ChunkGroups grp;
};
__device__ __forceinline__ bool chunk_lane64(ChunkLane64& L, const uint32_t* order, int n, int chunk, const double* st,
                                             size_t np, const GridGeom& g) {
    const int lane = threadIdx.x & 31, q0 = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * chunk;
    L.cnt = min(chunk, n - q0);
    if (L.cnt <= 0) return false;  // the whole warp
    L.valid = lane < L.cnt;
    L.p = (int)order[q0 + (L.valid ? lane : 0)];
#pragma unroll
    for (int c = 0; c < 3; c++) {
        const double x = st[(size_t)(PX + c) * np + L.p];
        L.base[c] = stencil_base<double>(x - g.mn[c], g.dx, g.dim[c]);
        axis_weights<double>(x, g.mn[c], g.dx, L.base[c], L.w[c], false);
    }
    L.grp = chunk_groups<false>(cell_key(L.base, g.dim), L.valid);
    return true;
}

// m_g += w m_p;  p_g += w (m_p v (1 - dt drag) + (-3/dx^2 dt vol P Fe^T + m_p C) (x_g - x_p))
// (SingleParticle_to_grid, ForwardSimulation.cpp:11-51)
static __global__ void __launch_bounds__(DMPM_CHUNK_THREADS, 4) k_p2g_c64(FwdArgs<double> a, const uint32_t* order, int chunk) {
    __shared__ __align__(16) double s_rec[DMPM_CHUNK_THREADS * kRec64];
    ChunkLane64 L;
    if (!chunk_lane64(L, order, a.n, chunk, a.st, a.np, a.geo)) return;
    double* rec = s_rec + (threadIdx.x & ~31) * kRec64;
    if (L.valid) {
        const int p = L.p;
        const double dx = a.geo.dx, mp = a.cst[(size_t)KM * a.np + p], damp = 1.0 - a.dt * a.drag;
        const m3<double> Fe = load_m3(a.st + (size_t)PF * a.np, a.np, p) + load_m3(a.dfc, a.np, p);
        const double k = -3.0 / (dx * dx) * a.dt * a.cst[(size_t)KVOL * a.np + p];
        const m3<double> G = (k * load_m3((const double*)a.P, a.np, p)) * transpose(Fe) +
                             mp * load_m3(a.st + (size_t)PC * a.np, a.np, p);
        double b[4];
#pragma unroll
        for (int c = 0; c < 3; c++) b[c] = mp * a.st[(size_t)(PV + c) * a.np + p] * damp;
        b[3] = mp;
        chunk_record64(rec + L.grp.slot * kRec64, L.w, b, G);
    }
    __syncwarp();
    chunk_scatter64<4>(rec, L.base, L.grp, a.geo, a.grid);
}
// dLdv_g += w dLdv_next + 3/dx^2 w dLdC_next (x_g - x_p)   (BackPropagation.cpp:27-44)
template <bool EXACT>
__global__ void __launch_bounds__(DMPM_CHUNK_THREADS, 4) k_adj_scatter_c64(AdjArgs<double> a, const uint32_t* order, int chunk) {
    __shared__ __align__(16) double s_rec[DMPM_CHUNK_THREADS * kRec64];
    ChunkLane64 L;
    if (!chunk_lane64(L, order, a.n, chunk, a.st, a.np, a.geo)) return;
    double* rec = s_rec + (threadIdx.x & ~31) * kRec64;
    if (L.valid) {
        const int p = L.p;
        const m3<double> Fe = load_m3(a.st + (size_t)PF * a.np, a.np, p) + load_m3(a.dfc, a.np, p);
        double b[4];
        m3<double> Cn;
        adj_next_terms<double, EXACT>(a, p, Fe, b, Cn);
        b[3] = 0.0;
        if (a.dbg_vnext) {
#pragma unroll
            for (int c = 0; c < 3; c++) a.dbg_vnext[(size_t)c * a.np + p] = b[c];
            store_m3(a.dbg_Cnext, a.np, p, Cn);
        }
        chunk_record64(rec + L.grp.slot * kRec64, L.w, b, (3.0 / (a.geo.dx * a.geo.dx)) * Cn);
    }
    __syncwarp();
    chunk_scatter64<3>(rec, L.base, L.grp, a.geo, a.gadj);
}

}  // namespace dmpm
