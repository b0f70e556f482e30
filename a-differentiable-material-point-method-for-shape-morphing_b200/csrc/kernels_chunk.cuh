// kernels_chunk.cuh -- FP32 path scatters over chunks of the sorted order.
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
    float* rec = s_rec + (threadIdx.x & ~31) * kRecFloats;
    float t[3];
    int base[3];
    load_x_base(a.st, a.npl, L.p, chunk_geo<BATCH>(a, L.inst), t, base, a.xlo);
    const ChunkGroups grp = chunk_groups<GENERAL>(chunk_key<BATCH>(a, L.inst, base), L.valid);
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
// 12.3; 79k 20.5 / 17.2 / 16.6 and 24.4 / 20.9 / 18.6; 267k 43.9 / 32.5 / 29.0
// and 58.3 / 43.4 / 39.8.  So: the most that leave 8 warps for each of 148 SMs.
inline int scatter_chunk(int n) {
    const int warps = 148 * 8;
    return n >= 32 * warps ? 32 : n >= 16 * warps ? 16 : 8;
}
// blocks of a chunk kernel over n particles, chunk particles a warp
inline unsigned chunk_blocks(int n, int chunk) {
    const int per = chunk * (DMPM_CHUNK_THREADS / 32);
    return (unsigned)((n + per - 1) / per);
}

}  // namespace dmpm
