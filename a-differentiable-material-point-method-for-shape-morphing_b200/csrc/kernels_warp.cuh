// kernels_warp.cuh -- FP32 path: what its kernels share (WArgs, the stress and
// finalize arithmetic, node passes and node boxes) and the deterministic mode's P2G
// and adjoint scatter over cell-sorted warp items.  The float mode's stencil kernels
// are in kernels_chunk.cuh.
//
// GENERAL (a test switch) forces the per-lane reductions everywhere.
//
// A warp item is a run of at most 8 particles that share a cell in the sorted
// order (sort.cuh).  One warp serves one item: lane = 4 q + s handles particle
// slot q (0..7) and stencil slab s (0..3), i.e. the 16 nodes
// (base_x + s, base_y + j, base_z + k), j, k in 0..3, fully unrolled with
// compile-time j, k.  When all 8 particles of the warp share the cell (the
// common case), the scatters combine the 8 particles' contributions with a
// butterfly reduce-scatter over the lanes of equal s, so each lane ends up
// owning one node's complete sum and adds it once, as integers (fixpoint.cuh);
// otherwise every lane adds its own.  The FP64 polar decomposition is
// stress_particle's (k_stress, or G2P for the next step) and finalize_particle's
// (the gather).
//
// Math per stage is that of kernels.cuh (which cites the reference).
//
// Strain storage: the FP32 path keeps each layer's deformation gradient as its
// strain H = F - I in the F planes (PF).  Strains of a few 1e-3 keep float's
// full relative precision this way, where F itself (about 1) would round them
// to ~1e-4 relative at every step.  Kernels form F = I + H where they need it
// -- in FP64 for the polar decomposition -- and update H directly:
//   H' = (1 - s)(D + dt C' (I + D)) + s H,  D = H + dFc.
// The host converts at upload and download; the FP64 path stores F.
#pragma once
#include "fixpoint.cuh"
#include "sort.cuh"

namespace dmpm {

// F + dFc = I + H + dFc of layer n, in float and (exactly) in double
__device__ __forceinline__ m3<float> fe_from_strain(const m3<float>& H, const m3<float>& dfc) {
    m3<float> r = H + dfc;
    r.a[0][0] += 1.f;
    r.a[1][1] += 1.f;
    r.a[2][2] += 1.f;
    return r;
}
__device__ __forceinline__ m3<double> fe_from_strain_d(const m3<float>& H, const m3<float>& dfc) {
    m3<double> r;
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
        for (int j = 0; j < 3; j++) r.a[i][j] = (double)H.a[i][j] + (double)dfc.a[i][j] + (i == j ? 1.0 : 0.0);
    return r;
}

struct WarpItems {
    const uint32_t* order;       // sorted particle indices
    const uint32_t* item_start;  // n_items + 1 entries
};

struct ItemLane {
    int p;       // particle index (slot 0's particle for idle lanes)
    bool valid;  // lane carries a particle
    int q, s;
};

__device__ __forceinline__ ItemLane item_lane(const WarpItems& it, int item) {
    ItemLane r;
    const int lane = threadIdx.x & 31;
    r.q = lane >> 2;
    r.s = lane & 3;
    const uint32_t st = it.item_start[item];
    const uint32_t cnt = it.item_start[item + 1] - st;
    r.valid = (uint32_t)r.q < cnt;
    r.p = (int)it.order[st + (r.valid ? r.q : 0)];
    return r;
}

// true when every lane's stencil base equals lane 0's
__device__ __forceinline__ bool warp_uniform_base(const int b[3]) {
    const int b0 = __shfl_sync(0xffffffffu, b[0], 0), b1 = __shfl_sync(0xffffffffu, b[1], 0),
              b2 = __shfl_sync(0xffffffffu, b[2], 0);
    return __all_sync(0xffffffffu, b[0] == b0 && b[1] == b1 && b[2] == b2);
}

// Butterfly reduce-scatter over the 8 lanes that share lane & 3, for vectors
// whose 8 blocks of N/8 entries the lanes hold in a lane-permuted order: lane
// L's block b holds stencil node b ^ perm(L), perm(L) = 4 (L>>4 & 1) +
// 2 (L>>3 & 1) + (L>>2 & 1) (scatter_perm).  Then at every stage each lane
// keeps the lower half and sends the upper half -- the partner holds the same
// nodes there -- with no per-lane selects.  On return v[0 .. N/8) of lane L
// hold the sums of node perm(L)'s entries over the 8 lanes.
template <int N> __device__ __forceinline__ void reduce_scatter8(float (&v)[N]) {
#pragma unroll
    for (int i = 0; i < N / 2; i++) v[i] += __shfl_xor_sync(0xffffffffu, v[i + N / 2], 16);
#pragma unroll
    for (int i = 0; i < N / 4; i++) v[i] += __shfl_xor_sync(0xffffffffu, v[i + N / 4], 8);
#pragma unroll
    for (int i = 0; i < N / 8; i++) v[i] += __shfl_xor_sync(0xffffffffu, v[i + N / 8], 4);
}
// this lane's node permutation for reduce_scatter8: row bit (jp) and axis-2 bits (kp)
struct ScatterPerm {
    int jp, kp;
};
__device__ __forceinline__ ScatterPerm scatter_perm() {
    const int lane = threadIdx.x & 31;
    return ScatterPerm{(lane >> 4) & 1, ((lane >> 3) & 1) * 2 + ((lane >> 2) & 1)};
}

template <int N> __device__ __forceinline__ void reduce_slabs(float (&v)[N]) {
#pragma unroll
    for (int i = 0; i < N; i++) {
        v[i] += __shfl_xor_sync(0xffffffffu, v[i], 1);
        v[i] += __shfl_xor_sync(0xffffffffu, v[i], 2);
    }
}

__device__ __forceinline__ bool in_grid(const GridGeom& g, int i, int j, int k) {
    return i >= 0 && i < g.dim[0] && j >= 0 && j < g.dim[1] && k >= 0 && k < g.dim[2];
}
__device__ __forceinline__ size_t node_id(const GridGeom& g, int i, int j, int k) {
    return ((size_t)i * g.dim[1] + j) * g.dim[2] + k;
}

// Node addressing of a lane's 16 stencil nodes (base_x + s, base_y + j, base_z + k):
// node (j, k) = g00 + j * dim_z + k in 32-bit arithmetic (grids are limited to
// 2^31 nodes) and bit 4j + k of mask says whether that node lies in the grid.
// g00 may point outside the grid; it is only dereferenced under the mask.
struct LaneNodes {
    int g00, sj;
    unsigned mask;
};
__device__ __forceinline__ LaneNodes lane_nodes(const GridGeom& g, const int base[3], int s) {
    LaneNodes r;
    const int gi = base[0] + s;
    r.sj = g.dim[2];
    r.g00 = (gi * g.dim[1] + base[1]) * g.dim[2] + base[2];
    unsigned mj = 0, mk = 0;
#pragma unroll
    for (int t = 0; t < 4; t++) {
        mj |= ((unsigned)(base[1] + t) < (unsigned)g.dim[1]) ? (1u << t) : 0u;
        mk |= ((unsigned)(base[2] + t) < (unsigned)g.dim[2]) ? (1u << t) : 0u;
    }
    unsigned m = 0;
#pragma unroll
    for (int j = 0; j < 4; j++) m |= ((mj >> j) & 1u) ? (mk << (4 * j)) : 0u;
    r.mask = ((unsigned)gi < (unsigned)g.dim[0]) ? m : 0u;
    return r;
}

// Per-lane stencil weights: slab s of axis 0, all 4 nodes of axis 2.
struct LaneW {
    float d0, n0;
    float d2[4], n2[4];
};
// Branch-free cubic B-spline and slope (same piecewise polynomials as
// Interpolation.h:5-30, evaluated with selects so divergent lanes do not
// serialise).
__device__ __forceinline__ float bsp(float q) {
    const float a = fabsf(q);
    const float inner = (0.5f * a - 1.f) * a * a + 2.f / 3.f;
    const float t = 2.f - a;
    const float outer = t * t * t * (1.f / 6.f);
    return a < 1.f ? inner : (a < 2.f ? outer : 0.f);
}
__device__ __forceinline__ float bsp_slope(float q) {
    const float a = fabsf(q);
    const float inner = (1.5f * a - 2.f) * q;
    const float t = 2.f - a;
    const float outer = copysignf(0.5f * t * t, -q);  // (-a/2 + 2 - 2/a) q without the division
    return a < 1.f ? inner : (a < 2.f ? outer : 0.f);
}

// The 4 lanes of a particle (equal lane >> 2) each evaluate the weights of
// stencil node s on all three axes; axis-2 values of the other nodes come from
// the sibling lanes by shuffles (every lane of the warp must call this).  Axis 1
// is left to the caller: it gets this lane's own axis-1 offset and weight in own1
// and fetches row j's values with row_weights (two shuffles) when it reaches that
// row, so only one row's values are live at a time.  Fills d0, n0 and the axis-2
// arrays of w, the latter in the order of node k ^ kperm (reduce_scatter8's
// permutation).
__device__ __forceinline__ void lane_weights_k(const float t[3], const GridGeom& g, int s, LaneW& w, float own1[2],
                                               int kperm) {
    const float dx = (float)g.dx;
    float d[3], n[3];
#pragma unroll
    for (int c = 0; c < 3; c++) {
        const float q = (float)s - t[c];
        d[c] = q * dx;
        n[c] = bsp(q);
    }
    w.d0 = d[0];
    w.n0 = n[0];
    own1[0] = d[1];
    own1[1] = n[1];
    const int grp = (threadIdx.x & 31) & ~3;
#pragma unroll
    for (int t = 0; t < 4; t++) {  // entry t holds axis-2 node t ^ kperm
        w.d2[t] = __shfl_sync(0xffffffffu, d[2], grp + (t ^ kperm));
        w.n2[t] = __shfl_sync(0xffffffffu, n[2], grp + (t ^ kperm));
    }
}
// row j's axis-1 (offset, weight) from the lane of slab j; every lane must call it
__device__ __forceinline__ void row_weights(const float own1[2], int j, float& d1, float& n1) {
    const int src = ((threadIdx.x & 31) & ~3) + j;
    d1 = __shfl_sync(0xffffffffu, own1[0], src);
    n1 = __shfl_sync(0xffffffffu, own1[1], src);
}

// stencil base and lattice coordinates t = (x - mn) / dx - base of particle p
// (compensated positions when xlo: load_xd, stencil_coord); xd, if given,
// receives the positions
__device__ __forceinline__ void load_x_base(const float* st, size_t np, int p, const GridGeom& g, float t[3],
                                            int base[3], int xlo, double* xd = nullptr) {
    const double idx = 1.0 / g.dx;
#pragma unroll
    for (int c = 0; c < 3; c++) {
        const double x = load_xd(st, np, p, c, xlo);
        if (xd) xd[c] = x;
        t[c] = stencil_coord<float>(x, g.mn[c], idx, g.dim[c], base[c]);
    }
}
// x' = x + dt v of axis c from the position x read by load_x_base, into the
// next layer's planes (hi and, when xlo, lo); returns the stored hi
__device__ __forceinline__ float store_x(float* st_next, size_t npn, int p, int c, double x, float dt, float v,
                                         int xlo) {
    if (!xlo) {
        const float xn = (float)x + dt * v;
        st_next[(size_t)(PX + c) * npn + p] = xn;
        return xn;
    }
    const double xn = x + (double)(dt * v);
    const float hi = (float)xn;
    st_next[(size_t)(PX + c) * npn + p] = hi;
    st_next[(size_t)(PXL + c) * npn + p] = (float)(xn - (double)hi);
    return hi;
}
// ------------------------------------------------------------------ args
// Minimum resident blocks per SM (the register cap the compiler works to) for
// k_stress at 256 threads per block (2: 128 registers, no spills; 1 lets it take
// 132 and run one block per SM)
// k_stress takes the FP64 polar factors from the scaled Newton iteration
// (polar_newton) where det(F + dFc) > 0 and from the SVD (polar3) otherwise;
// 0 uses the SVD everywhere
#ifndef DMPM_NEWTON_POLAR
#define DMPM_NEWTON_POLAR 1
#endif
#ifndef DMPM_STRESS_MIN_BLOCKS
#define DMPM_STRESS_MIN_BLOCKS 2
#endif
// and for the warp-item kernels: P2G in blocks of DMPM_P2G_THREADS (256), the
// adjoint scatter below in blocks of DMPM_ADJ_SCATTER_THREADS (128)
#ifndef DMPM_SCATTER_MIN_BLOCKS
#define DMPM_SCATTER_MIN_BLOCKS 3
#endif
#ifndef DMPM_P2G_THREADS
#define DMPM_P2G_THREADS 256
#endif
// CTAs per SM of the persistent grids (no more than the register budget above lets reside)
#ifndef DMPM_SCATTER_CTAS
#define DMPM_SCATTER_CTAS DMPM_SCATTER_MIN_BLOCKS
#endif
// the adjoint scatter on its own, in blocks of 128 threads, 7 per SM (72 registers);
// measured when it also formed its sources and added floats: 53.3 us on the 64^3,
// 267k-particle scene against 55.4 us for 4 blocks of 256, 59.4 for 3 of 256 and
// 55.7 for 5 of 128; P2G was faster at 3 blocks of 256
#ifndef DMPM_ADJ_SCATTER_MIN_BLOCKS
#define DMPM_ADJ_SCATTER_MIN_BLOCKS 7
#endif
#ifndef DMPM_ADJ_SCATTER_THREADS
#define DMPM_ADJ_SCATTER_THREADS 128
#endif
#ifndef DMPM_ADJ_SCATTER_CTAS
#define DMPM_ADJ_SCATTER_CTAS DMPM_ADJ_SCATTER_MIN_BLOCKS
#endif

// Grid of one instance of a batch: its geometry, the offset of its first node
// in the batch's concatenated grids and of its first cell key.
struct InstGeo {
    GridGeom g;
    int goff;
    uint32_t koff;
};

// Plane strides: np for the per-particle constants, controls and adjoint
// scratch; npl for the state, affine/polar planes and adjoint of layer n;
// npn for the state and adjoint of layer n + 1.  One scene: all three equal.
// A batch stores each layer for the instances still running, so its layers
// have their own strides.
struct WArgs {
    int n;
    int chunk;             // particles per warp of the chunk kernels (kernels_chunk.cuh): 8, 16 or 32
    size_t np, npl, npn;
    GridGeom geo;
    float dt, drag, s, fext[3];
    WarpItems items;
    const uint32_t* n_items_dev;  // warp item count, on the device
    const InstGeo* ig;            // batch: per-instance grids
    const uint16_t* pinst;        // batch: instance of each particle
    const float* st;       // layer n state
    float* st_next;        // layer n+1 state
    int xlo;               // st and st_next carry the low parts of compensated positions (planes PXL)
    const float* cst;      // constants
    const float* dfc;      // dFc of layer n
    float* G;              // [24][npl] per layer: G (9), polar R (9), polar S (6: s00 s01 s02 s11 s12 s22)
    node4<float>* grid;    // layer n grid: (p, m) after P2G, (v, m) after the grid update
    int* box;              // node box that P2G widens to the stencils it adds to (NodeRange), or null
    int* box_next;         // G2P: the next layer's box, which takes in this one's, or null
    float* P;              // debug: stress of layer n (or null)
    unsigned* status;
    // adjoint
    const float* adj_next;
    float* adj;
    float* adjn;           // [12][np]: dLdv_next (3), dLdC_next (9)
    node4<float>* gadj;    // (dLdv.xyz, 0)
    node4<float>* gadj2;   // per node two records: (dLdp.xyz, dLdm), (v.xyz, m)
    float* ctrl_grad;      // per-layer dL/d dFc [9][np] or null
    double* ctrl_acc;      // tied FP64 accumulator or null
    float* dbg_dLdP;
    float* dbg_vnext;
    float* dbg_Cnext;
    // G2P with the next step's stress stage (kernels_chunk.cuh): dFc of layer n + 1,
    // its G planes and its debug P (or null)
    const float* dfc_next;
    float* G_next;
    float* P_next;
    int n_next;            // particles that take the next step (a batch's shorter rollouts end)
    // deterministic mode (fixpoint.cuh): integer node sums and their bound slots, or null
    fix4* fix;
    unsigned* fixb;
    // brick units of the sorted order (kernels_brick.cuh): unit u holds the
    // sorted positions [unit_start[u], unit_start[u + 1]), all with key >> shift
    // equal to unit_key[u]; the unit count stays on the device
    const uint32_t* unit_start;
    const uint32_t* unit_key;
    const uint32_t* n_units_dev;
    const uint32_t* unit_item;  // first warp item of each unit (n_units + 1 entries), or null
};

// Persistent launches over warp items: the item count stays on the device.
__device__ __forceinline__ int first_warp() { return (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5); }
__device__ __forceinline__ int warp_count() { return (int)((gridDim.x * blockDim.x) >> 5); }

// ------------------------------------------------------------------ forward
// P = PK(F + dFc) in FP64;  G = -3/dx^2 dt vol P Fe^T + m C  (P_op_1 and the
// particle-constant part of SingleParticle_to_grid, ForwardSimulation.cpp:6-9, 38)
// The stress stage of particle p: the FP64 polar decomposition of
// Fe = I + H + dFc (scaled Newton where det > 0, SVD otherwise), P, and
// G = -3/dx^2 dt vol P Fe^T + m C.  Writes G and the polar factors R, S (for
// the adjoint's k_adj_finalize) into the planes at Gp (stride ng) and P into Pp
// unless it is null; returns G.  cfetch() gives C, fetched after the polar so
// that it holds no registers through it.
template <class CFetch>
__device__ __forceinline__ m3<float> stress_particle(const WArgs& a, int p, const m3<float>& H, const m3<float>& dfc,
                                                     const CFetch& cfetch, float* Gp, size_t ng, float* Pp) {
    const size_t np = a.np;
    const m3<float> Fe = fe_from_strain(H, dfc);
    const m3<double> Fed = fe_from_strain_d(H, dfc);
    m3<double> Rd, Sd;
    if (!DMPM_NEWTON_POLAR || !polar_newton(Fed, Rd, Sd)) polar3(Fed, Rd, Sd);
    const m3<double> Pd = pk_from_polar(Fed, Rd, (double)a.cst[(size_t)KLAM * np + p], (double)a.cst[(size_t)KMU * np + p]);
    const m3<float> P = m3_cast<float>(Pd);
    if (Pp) store_m3(Pp, ng, p, P);
    store_m3(Gp + 9 * ng, ng, p, m3_cast<float>(Rd));
    Gp[18 * ng + p] = (float)Sd.a[0][0];
    Gp[19 * ng + p] = (float)Sd.a[0][1];
    Gp[20 * ng + p] = (float)Sd.a[0][2];
    Gp[21 * ng + p] = (float)Sd.a[1][1];
    Gp[22 * ng + p] = (float)Sd.a[1][2];
    Gp[23 * ng + p] = (float)Sd.a[2][2];
    const float dx = (float)a.geo.dx;
    const float k = -3.f / (dx * dx) * a.dt * a.cst[(size_t)KVOL * np + p];
    const m3<float> G = (k * P) * transpose(Fe) + a.cst[(size_t)KM * np + p] * cfetch();
    store_m3(Gp, ng, p, G);
    return G;
}

// DET: also raise the deterministic mode's P2G bounds (fixpoint.cuh) in a.fixb.
template <bool DET = false> __global__ void __launch_bounds__(256, DMPM_STRESS_MIN_BLOCKS) k_stress(WArgs a) {
    const size_t np = a.np, npl = a.npl;
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    float cmom = 0.f, cmass = 0.f;
    if (p < a.n) {
        const m3<float> H = load_m3(a.st + (size_t)PF * npl, npl, p), dfc = load_m3(a.dfc, np, p);
        const m3<float> G = stress_particle(
            a, p, H, dfc, [&]() { return load_m3(a.st + (size_t)PC * npl, npl, p); }, a.G, npl, a.P);
        if constexpr (DET) {
            const float dx = (float)a.geo.dx;
            // bound on P2G's per-particle values: |m v damp + G d| with |d| < 2 dx, and m
            const float mp = a.cst[(size_t)KM * np + p], damp = 1.f - a.dt * a.drag;
#pragma unroll
            for (int c = 0; c < 3; c++) {
                const float t = fabsf(mp * a.st[(size_t)(PV + c) * npl + p] * damp) +
                                2.f * dx * (fabsf(G.a[c][0]) + fabsf(G.a[c][1]) + fabsf(G.a[c][2]));
                cmom = fmaxf(cmom, t);
            }
            cmass = mp;
        }
    }
    if constexpr (DET) {  // every lane of every warp reaches these
        fix_bound(a.fixb + FIXB_MOMENTUM, cmom * 1.001f);
        fix_bound(a.fixb + FIXB_MASS, cmass * 1.001f);
    }
}

// P2G: m_g += w m_p;  p_g += w (m_p v (1 - dt drag) + G (x_g - x_p))
// One warp item of P2G in the deterministic mode: integer node sums
// (fixpoint.cuh) into a.fix, or with a tile (ft.t non-null) those of an item
// whose stencil lies in the tile into its shared-memory integers.
template <bool GENERAL, bool TILE>
__device__ __forceinline__ void p2g_item(const WArgs& a, int item, const FixScale& sp, const FixScale& sm,
                                         const FixTile& ft) {
    const size_t np = a.np, npl = a.npl;
    {
        const GridGeom& geo = a.geo;
        const ItemLane L = item_lane(a.items, item);
        float t[3];
        int base[3];
        load_x_base(a.st, npl, L.p, geo, t, base, a.xlo);
        const bool uniform = !GENERAL && warp_uniform_base(base);
        // slot (jj, kk) of each half holds node (2 half + (jj ^ P.jp), kk ^ P.kp)
        const ScatterPerm P = scatter_perm();
        LaneW w;
        float own1[2];
        lane_weights_k(t, geo, L.s, w, own1, P.kp);
        const float mp = L.valid ? a.cst[(size_t)KM * np + L.p] : 0.f;
        const float damp = 1.f - a.dt * a.drag;
        float mvd[3], g0[3];
        m3<float> G = load_m3(a.G, npl, L.p);
#pragma unroll
        for (int c = 0; c < 3; c++) {
            mvd[c] = mp * a.st[(size_t)(PV + c) * npl + L.p] * damp;
            g0[c] = G.a[c][0] * w.d0;
        }
        const LaneNodes N = lane_nodes(geo, base, L.s);
        // tile offset of node (0, 0, 0) of the item's stencil, or -1 when the stencil is not inside the tile
        const int tile_l = TILE && uniform ? fix_tile_offset(ft, base) : -1;
#pragma unroll
        for (int half = 0; half < 2; half++) {
            float v[32];
#pragma unroll
            for (int jj = 0; jj < 2; jj++) {
                float d1, n1;
                row_weights(own1, 2 * half + (jj ^ P.jp), d1, n1);
                float g1[3];
#pragma unroll
                for (int c = 0; c < 3; c++) g1[c] = g0[c] + G.a[c][1] * d1;
                const float w01 = L.valid ? w.n0 * n1 : 0.f;
#pragma unroll
                for (int kk = 0; kk < 4; kk++) {
                    const float wt = w01 * w.n2[kk];
                    const int o = (jj * 4 + kk) * 4;
#pragma unroll
                    for (int c = 0; c < 3; c++) v[o + c] = wt * (mvd[c] + g1[c] + G.a[c][2] * w.d2[kk]);
                    v[o + 3] = wt * mp;
                }
            }
            if (uniform) {
                reduce_scatter8<32>(v);
                const int j = 2 * half + P.jp, k = P.kp;
                if (((N.mask >> (4 * j + k)) & 1u) && (v[0] != 0.f || v[1] != 0.f || v[2] != 0.f || v[3] != 0.f)) {
                    if (TILE && tile_l >= 0)
                        fix_red4_tile(ft, tile_l + (L.s * ft.E + j) * ft.E + k, v[0], v[1], v[2], v[3], sp.s, sm.s);
                    else
                        fix_red4(a.fix + (N.g00 + j * N.sj + k), v[0], v[1], v[2], v[3], sp.s, sm.s);
                }
            } else if (L.valid) {
#pragma unroll
                for (int nd = 0; nd < 8; nd++) {
                    const int j = 2 * half + ((nd >> 2) ^ P.jp), k = (nd & 3) ^ P.kp;
                    if (!((N.mask >> (4 * j + k)) & 1u)) continue;
                    fix_red4(a.fix + (N.g00 + j * N.sj + k), v[nd * 4], v[nd * 4 + 1], v[nd * 4 + 2], v[nd * 4 + 3],
                             sp.s, sm.s);
                }
            }
        }
    }
}

// P2G over warp items (one item per warp, persistent grid-stride)
template <bool GENERAL> __global__ void __launch_bounds__(DMPM_P2G_THREADS, DMPM_SCATTER_MIN_BLOCKS) k_p2g_w(WArgs a) {
    const int nit = (int)*a.n_items_dev;
    const FixScale sp = fix_scale(a.fixb + FIXB_MOMENTUM, a.n), sm = fix_scale(a.fixb + FIXB_MASS, a.n);
    const FixTile none{nullptr, 0, {0, 0, 0}, 0};
    for (int item = first_warp(); item < nit; item += warp_count()) p2g_item<GENERAL, false>(a, item, sp, sm, none);
}

// G_op in place: (p, m) -> (v, m), v = p/m + dt f where |m| > FLT_EPSILON, else 0
__device__ __forceinline__ void gop_node(node4<float>* n, float dt, const float f[3]) {
    node4<float> nd = *n;
    float v[3];
    node_velocity(nd, dt, f, v);
    nd.x = v[0];
    nd.y = v[1];
    nd.z = v[2];
    *n = nd;
}
static __global__ void k_gop_inplace(node4<float>* grid, size_t G, float dt, float f0, float f1, float f2) {
    const size_t g = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= G) return;
    const float f[3] = {f0, f1, f2};
    gop_node(grid + g, dt, f);
}

// Node boxes.  A cloud fills a part of its grid: 8 % of the 64^3 headline scene's
// nodes, 3 % of a 256^3 grid with a sphere of 79 cells.  Each layer's grid has a box
// of nodes (first and last per axis, 6 ints) outside which it is zero, and the
// node passes of the layer -- clearing its grid before P2G, the grid update, the
// adjoint grid update -- walk the box instead of the grid.  P2G widens the box to
// the stencils it adds to; boxes only grow (until a new cloud is set up), and a
// layer's takes in the layer's before it first (in G2P, once the grid is cleared),
// so that P2G finds it wide enough nearly always and few warps reach the atomics
// (starting empty at every step,
// P2G took 55 instead of 29 us per step on the 64^3, 267k-particle scene).
// One warp walks a row of the box along the last axis.
struct NodeRange {
    int lo[3], n[3];
    __device__ __forceinline__ NodeRange(const int* box) {
#pragma unroll
        for (int c = 0; c < 3; c++) {
            lo[c] = box[c];
            n[c] = box[3 + c] - box[c] + 1;  // <= 0: empty
        }
    }
    __device__ __forceinline__ int rows() const { return n[0] > 0 && n[1] > 0 && n[2] > 0 ? n[0] * n[1] : 0; }
    __device__ __forceinline__ size_t first(int row, const GridGeom& g) const {
        const int i = row / n[1];
        return node_id(g, lo[0] + i, lo[1] + (row - i * n[1]), lo[2]);
    }
};
constexpr int kEmptyLo = 0x7fffffff;
// boxes [0, grids) empty, box `grids` the whole grid
static __global__ void k_box_reset(int* boxes, int grids, GridGeom g) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x, b = t / 6, c = t % 6;
    if (b > grids) return;
    boxes[t] = b == grids ? (c < 3 ? 0 : g.dim[c - 3] - 1) : (c < 3 ? kEmptyLo : -1);
}
// every lane of the warp: widen the box to the stencils of the valid lanes; have:
// lanes 0..5 the box's ints as read when the kernel began
__device__ __forceinline__ void widen_box(int* box, int have, const GridGeom& g, const int base[3], bool valid) {
    const int lane = threadIdx.x & 31;
    int lo = kEmptyLo, hi = -1;  // of axis lane (lo) and lane - 3 (hi)
    bool some = true;            // the warp has a node inside the grid
#pragma unroll
    for (int c = 0; c < 3; c++) {
        const int l = max(0, __reduce_min_sync(0xffffffffu, valid ? base[c] : kEmptyLo));
        const int h = min(g.dim[c] - 1, __reduce_max_sync(0xffffffffu, valid ? base[c] + 3 : -1));
        some &= l <= h;
        lo = lane == c ? l : lo;
        hi = lane == 3 + c ? h : hi;
    }
    if (!some) return;
    if (lane < 3 && lo < have) atomicMin(box + lane, lo);
    if (lane >= 3 && lane < 6 && hi > have) atomicMax(box + lane, hi);
}
// the same for the positions of a layer state
static __global__ void __launch_bounds__(256) k_box_points(const float* st, size_t np, int n, GridGeom g, int* box) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    float t[3];
    int base[3];
    load_x_base(st, np, min(p, n - 1), g, t, base, 1);
    widen_box(box, (threadIdx.x & 31) < 6 ? *(volatile int*)(box + (threadIdx.x & 31)) : 0, g, base, p < n);
}
// zero the nodes of the layer's box.  Nothing may write the box meanwhile: the rows
// are numbered by it, and a warp that saw another box would leave rows to nobody.
__device__ __forceinline__ void box_clear(node4<float>* grid, const int* box, const GridGeom& g) {
    const NodeRange r(box);
    for (int row = first_warp(); row < r.rows(); row += warp_count()) {
        node4<float>* p = grid + r.first(row, g);
        for (int k = threadIdx.x & 31; k < r.n[2]; k += 32) p[k] = node4<float>{0.f, 0.f, 0.f, 0.f};
    }
}
static __global__ void __launch_bounds__(256) k_box_clear(node4<float>* grid, const int* __restrict__ box, GridGeom g) {
    box_clear(grid, box, g);
}
// lanes 0..5 of one warp of G2P, between the clearing of the next layer's grid and
// its P2G: the next layer's box takes in this one's
__device__ __forceinline__ void box_join(int* next, const int* box) {
    const int c = threadIdx.x;
    if (c < 6) next[c] = c < 3 ? min(next[c], box[c]) : max(next[c], box[c]);
}
// the grid update over the box; next: the next layer's grid, cleared as by
// k_box_clear for a launch less per step (8.7k particles: 39.9 -> 38.7 us a step
// forward and back), or null
static __global__ void __launch_bounds__(256)
    k_box_gop(node4<float>* grid, const int* __restrict__ box, node4<float>* next, const int* __restrict__ next_box,
              GridGeom g, float dt, float f0, float f1, float f2) {
    const NodeRange r(box);
    if (next) box_clear(next, next_box, g);
    const float f[3] = {f0, f1, f2};
    for (int row = first_warp(); row < r.rows(); row += warp_count()) {
        node4<float>* p = grid + r.first(row, g);
        for (int k = threadIdx.x & 31; k < r.n[2]; k += 32) gop_node(p + k, dt, f);
    }
}

// The deterministic mode's: integer sums to (p, m) to (v, m) over the whole grid,
// whose box becomes the layer's.  Bound by the 32 + 16 bytes per node.  As a memset
// of the sums, a conversion and a grid update 34 us per step forward and back
// on a 64 x 60 x 53 grid; this and k_fix_adj_gop, 17.
static __global__ void __launch_bounds__(256)
    k_fix_gop(fix4* acc, const unsigned* __restrict__ slots, long long n, size_t G, node4<float>* grid,
              const int* __restrict__ whole, int* box, float dt, float f0, float f1, float f2) {
    const size_t g = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (g < 6) box[g] = whole[g];
    if (g >= G) return;
    const float f[3] = {f0, f1, f2};
    node4<float> nd = fix_take(acc + g, slots, n, 0);
    gop_node(&nd, dt, f);
    grid[g] = nd;
}

// ------------------------------------------------------------------ adjoint
// dLdv_next = dt dLdx' + dLdv';  dLdC_next = c dt dLdF' Fe^T + dLdC'
// dLdv_g += w dLdv_next + 3/dx^2 w dLdC_next (x_g - x_p)   (BackPropagation.cpp:14-44)
// The per-particle sources of the adjoint scatter: vn = dt dLdx' + dLdv' and
// Cn = cf dLdF' Fe^T + dLdC' (cf = (1 - s) dt exact, dt refcompat), from layer
// n + 1's adjoint and layer n's F + dFc.
template <bool EXACT>
__device__ __forceinline__ void adj_sources(const WArgs& a, int p, float vn[3], m3<float>& Cn) {
    const size_t np = a.np, npl = a.npl, npn = a.npn;
#pragma unroll
    for (int c = 0; c < 3; c++) vn[c] = a.dt * a.adj_next[(size_t)(PX + c) * npn + p] + a.adj_next[(size_t)(PV + c) * npn + p];
    const m3<float> Fe = fe_from_strain(load_m3(a.st + (size_t)PF * npl, npl, p), load_m3(a.dfc, np, p));
    const float cf = EXACT ? (1.f - a.s) * a.dt : a.dt;
    Cn = (cf * load_m3(a.adj_next + (size_t)PF * npn, npn, p)) * transpose(Fe) +
         load_m3(a.adj_next + (size_t)PC * npn, npn, p);
}

// Deterministic mode: the scatter's sources per particle into adjn (which the
// gather reads too) and their bound |vn + 3/dx^2 Cn d| with |d| < 2 dx into
// the adjoint bound slot, before the scatter adds anything.
template <bool EXACT> __global__ void __launch_bounds__(256) k_adj_sources(WArgs a) {
    const size_t np = a.np;
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    float c = 0.f;
    if (p < a.n) {
        float vn[3];
        m3<float> Cn;
        adj_sources<EXACT>(a, p, vn, Cn);
#pragma unroll
        for (int r = 0; r < 3; r++) a.adjn[(size_t)r * np + p] = vn[r];
        store_m3(a.adjn + 3 * np, np, p, Cn);
        if (a.dbg_vnext) {
#pragma unroll
            for (int r = 0; r < 3; r++) a.dbg_vnext[(size_t)r * np + p] = vn[r];
        }
        if (a.dbg_Cnext) store_m3(a.dbg_Cnext, np, p, Cn);
        const float dx = (float)a.geo.dx, k3 = 3.f / (dx * dx);
#pragma unroll
        for (int r = 0; r < 3; r++)
            c = fmaxf(c, fabsf(vn[r]) + k3 * 2.f * dx * (fabsf(Cn.a[r][0]) + fabsf(Cn.a[r][1]) + fabsf(Cn.a[r][2])));
    }
    fix_bound(a.fixb + FIXB_ADJ, c * 1.001f);
}

// Warp items first, first + stride, ... below end of the deterministic mode's
// adjoint scatter: the sources come from k_adj_sources (adjn), the node sums go
// to a.fix as integers (fixpoint.cuh) or, with a tile, those of an item whose
// stencil lies in it to the tile's shared-memory integers.
template <bool GENERAL, bool TILE>
__device__ __forceinline__ void adj_scatter_items(const WArgs& a, int first, int end, int stride, const FixScale& sa,
                                                  const FixTile& ft) {
    const size_t np = a.np, npl = a.npl;
    for (int item = first; item < end; item += stride) {
        const GridGeom& geo = a.geo;
        const ItemLane L = item_lane(a.items, item);
        const int p = L.p;
        float t[3];
        int base[3];
        load_x_base(a.st, npl, p, geo, t, base, a.xlo);
        const bool uniform = !GENERAL && warp_uniform_base(base);
        const ScatterPerm P = scatter_perm();  // as in p2g_item
        LaneW w;
        float own1[2];
        lane_weights_k(t, geo, L.s, w, own1, P.kp);
        float vn[3];
#pragma unroll
        for (int c = 0; c < 3; c++) vn[c] = a.adjn[(size_t)c * np + p];
        const m3<float> Cn = load_m3(a.adjn + 3 * np, np, p);
        const float dx = (float)geo.dx;
        const float k3 = 3.f / (dx * dx);
        float c0[3];
#pragma unroll
        for (int r = 0; r < 3; r++) c0[r] = k3 * Cn.a[r][0] * w.d0;
        const LaneNodes N = lane_nodes(geo, base, L.s);
        const int tile_l = TILE && uniform ? fix_tile_offset(ft, base) : -1;
#pragma unroll
        for (int half = 0; half < 2; half++) {
            float v[24];  // 8 nodes x dLdv_g (3)
#pragma unroll
            for (int jj = 0; jj < 2; jj++) {
                float d1, n1;
                row_weights(own1, 2 * half + (jj ^ P.jp), d1, n1);
                float c1[3];
#pragma unroll
                for (int r = 0; r < 3; r++) c1[r] = c0[r] + k3 * Cn.a[r][1] * d1;
                const float w01 = L.valid ? w.n0 * n1 : 0.f;
#pragma unroll
                for (int kk = 0; kk < 4; kk++) {
                    const float wt = w01 * w.n2[kk];
                    const int o = (jj * 4 + kk) * 3;
#pragma unroll
                    for (int r = 0; r < 3; r++) v[o + r] = wt * (vn[r] + c1[r] + k3 * Cn.a[r][2] * w.d2[kk]);
                }
            }
            if (uniform) {
                reduce_scatter8<24>(v);
                const int j = 2 * half + P.jp, k = P.kp;
                if (((N.mask >> (4 * j + k)) & 1u) && (v[0] != 0.f || v[1] != 0.f || v[2] != 0.f)) {
                    if (TILE && tile_l >= 0)
                        fix_red4_tile(ft, tile_l + (L.s * ft.E + j) * ft.E + k, v[0], v[1], v[2], 0.f, sa.s, sa.s);
                    else
                        fix_red4(a.fix + (N.g00 + j * N.sj + k), v[0], v[1], v[2], 0.f, sa.s, sa.s);
                }
            } else if (L.valid) {
#pragma unroll
                for (int nd = 0; nd < 8; nd++) {
                    const int j = 2 * half + ((nd >> 2) ^ P.jp), k = (nd & 3) ^ P.kp;
                    if (!((N.mask >> (4 * j + k)) & 1u)) continue;
                    fix_red4(a.fix + (N.g00 + j * N.sj + k), v[nd * 3], v[nd * 3 + 1], v[nd * 3 + 2], 0.f, sa.s, sa.s);
                }
            }
        }
    }
}

// adjoint scatter over warp items (one item per warp, persistent grid-stride)
template <bool GENERAL>
__global__ void __launch_bounds__(DMPM_ADJ_SCATTER_THREADS, DMPM_ADJ_SCATTER_MIN_BLOCKS) k_adj_scatter_w(WArgs a) {
    const FixScale sa = fix_scale(a.fixb + FIXB_ADJ, a.n);
    const FixTile none{nullptr, 0, {0, 0, 0}, 0};
    adj_scatter_items<GENERAL, false>(a, first_warp(), (int)*a.n_items_dev, warp_count(), sa, none);
}

// adjoint G_op per node: (dLdp, dLdm) from dLdv and the layer's (v, m)
// The record pair (dLdp, dLdm), (v, m) of a node is stored contiguously (32 B)
// so the gather reads one sector per node.
template <bool EXACT>
__device__ __forceinline__ void adj_gop_node(const node4<float>& nd, const node4<float>& dv, node4<float>* out, float dt,
                                             const float f[3]) {
    node4<float> o{0.f, 0.f, 0.f, 0.f};
    if (fabsf(nd.w) > (float)kFltEps) {
        float v[3] = {nd.x, nd.y, nd.z};
        if (EXACT) { v[0] -= dt * f[0]; v[1] -= dt * f[1]; v[2] -= dt * f[2]; }
        o.x = dv.x / nd.w;
        o.y = dv.y / nd.w;
        o.z = dv.z / nd.w;
        o.w = -1.f / nd.w * (v[0] * dv.x + v[1] * dv.y + v[2] * dv.z);
    }
    out[0] = o;
    out[1] = nd;
}
template <bool EXACT>
__global__ void k_adj_gop_w(const node4<float>* __restrict__ grid, const node4<float>* __restrict__ gadj,
                            node4<float>* gadj2, size_t G, float dt, float f0, float f1, float f2) {
    const size_t g = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= G) return;
    const float f[3] = {f0, f1, f2};
    adj_gop_node<EXACT>(grid[g], gadj[g], gadj2 + 2 * g, dt, f);
}
// the same over the layer's box, clearing dLdv behind it for the next scatter
template <bool EXACT>
__global__ void __launch_bounds__(256)
    k_box_adj_gop(const node4<float>* __restrict__ grid, node4<float>* gadj, node4<float>* gadj2,
                  const int* __restrict__ box, GridGeom g, float dt, float f0, float f1, float f2) {
    const NodeRange r(box);
    const float f[3] = {f0, f1, f2};
    for (int row = first_warp(); row < r.rows(); row += warp_count()) {
        const size_t n0 = r.first(row, g);
        for (int k = threadIdx.x & 31; k < r.n[2]; k += 32) {
            adj_gop_node<EXACT>(grid[n0 + k], gadj[n0 + k], gadj2 + 2 * (n0 + k), dt, f);
            gadj[n0 + k] = node4<float>{0.f, 0.f, 0.f, 0.f};
        }
    }
}

// the deterministic mode's, from the integer sums of dLdv over the whole grid
template <bool EXACT>
__global__ void __launch_bounds__(256)
    k_fix_adj_gop(fix4* acc, const unsigned* __restrict__ slots, long long n, size_t G, const node4<float>* __restrict__ grid,
                  node4<float>* gadj2, float dt, float f0, float f1, float f2) {
    const size_t g = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= G) return;
    const float f[3] = {f0, f1, f2};
    adj_gop_node<EXACT>(grid[g], fix_take(acc + g, slots, n, 1), gadj2 + 2 * g, dt, f);
}

// ------------------------------------------------------------------ finalize
// per particle: P, polar factors and dP/dF in FP64, then the adjoint of layer n
//   dLdP = -3/dx^2 dt vol M^T Fe,  dLdF(stress) = -3/dx^2 dt vol M P,  dLdC = m M^T
//   dLdx = -X/dx - G^T u - 3/dx^2 dLdC_next^T z + dLdx',  dLdv = m (1 - dt drag) u
//   REFCOMPAT: dLdF = (1-s)T + s dLdF' + stress + T + dP:dLdP,  T = (I + dt C')^T dLdF'
//   EXACT:     dLdFe = (1-s)T + stress + dP:dLdP,  dLdF = dLdFe + s dLdF'
//
// Its inputs are 94 floats per particle (slots below), of which the gather's 18 sums
// are in registers and 18 are staged in shared memory by then, the rest in planes,
// and, with tied controls, the 9 FP64 planes of the control-gradient accumulator.
enum : int {
    FS_GATH = 0,    // 18: M (9, row-major), X (3), u (3), z (3)
    FS_F = 18,      // 9: strain H = F - I of layer n
    FS_DFC = 27,    // 9: dFc
    FS_AUX = 36,    // 24: G (9), polar R (9), polar S (6)
    FS_CST = 60,    // 4: m, vol, lam, mu
    FS_CN = 64,     // 9: dLdC_next
    FS_AX = 73,     // 3: dLdx of layer n+1
    FS_AF = 76,     // 9: dLdF of layer n+1
    FS_CNEXT = 85,  // 9: C of layer n+1
    FS_COUNT = 94
};

// first element and stride of a slot's plane (the sums of FS_GATH have none)
__device__ __forceinline__ const float* fin_plane(const WArgs& a, int slot, size_t& stride) {
    if (slot < FS_DFC) { stride = a.npl; return a.st + (size_t)(PF + slot - FS_F) * a.npl; }
    if (slot < FS_AUX) { stride = a.np; return a.dfc + (size_t)(slot - FS_DFC) * a.np; }
    if (slot < FS_CST) { stride = a.npl; return a.G + (size_t)(slot - FS_AUX) * a.npl; }
    if (slot < FS_CN) { stride = a.np; return a.cst + (size_t)(slot - FS_CST) * a.np; }
    if (slot < FS_AX) { stride = a.np; return a.adjn + (size_t)(3 + slot - FS_CN) * a.np; }
    if (slot < FS_AF) { stride = a.npn; return a.adj_next + (size_t)(PX + slot - FS_AX) * a.npn; }
    if (slot < FS_CNEXT) { stride = a.npn; return a.adj_next + (size_t)(PF + slot - FS_AF) * a.npn; }
    stride = a.npn;
    return a.st_next + (size_t)(PC + slot - FS_CNEXT) * a.npn;
}

template <bool EXACT, class In> __device__ __forceinline__ void finalize_particle(const WArgs& a, int p, const In& in) {
    const size_t np = a.np, npl = a.npl;
    auto mat = [&](int slot) {  // 9 column-major planes -> m3
        m3<float> m;
#pragma unroll
        for (int r = 0; r < 3; r++)
#pragma unroll
            for (int c = 0; c < 3; c++) m.a[r][c] = in(slot + r + 3 * c);
        return m;
    };
    m3<float> M;
#pragma unroll
    for (int r = 0; r < 3; r++)
#pragma unroll
        for (int c = 0; c < 3; c++) M.a[r][c] = in(FS_GATH + 3 * r + c);
    const float dx = (float)a.geo.dx;
    const float k3 = 3.f / (dx * dx);
    // dLdx = -X/dx - G^T u - 3/dx^2 dLdC_next^T z + dLdx',  dLdv = m (1 - dt drag) u,  dLdC = m M^T
    auto transport = [&]() {
        const float mp = in(FS_CST + KM);
        const m3<float> G = mat(FS_AUX);
        const m3<float> Cn = mat(FS_CN);
        float u[3], z[3], gtu[3], ctz[3];
#pragma unroll
        for (int c = 0; c < 3; c++) {
            u[c] = in(FS_GATH + 12 + c);
            z[c] = in(FS_GATH + 15 + c);
        }
        mtv(G, u, gtu);
        mtv(Cn, z, ctz);
        float ax0 = 0.f;
#pragma unroll
        for (int c = 0; c < 3; c++) {
            const float X = in(FS_GATH + 9 + c);
            const float ax = -X / dx - gtu[c] - k3 * ctz[c] + in(FS_AX + c);
            if (c == 0) ax0 = ax;
            a.adj[(size_t)(PX + c) * npl + p] = ax;
            a.adj[(size_t)(PV + c) * npl + p] = mp * (1.f - a.dt * a.drag) * u[c];
        }
        store_m3(a.adj + (size_t)PC * npl, npl, p, mp * transpose(M));
        return ax0;
    };
    const m3<float> H = mat(FS_F), dfc = mat(FS_DFC);
    const m3<float> Fe = fe_from_strain(H, dfc);
    const m3<double> Fed = fe_from_strain_d(H, dfc);
    // polar factors computed in FP64 by k_stress for this layer
    const m3<double> Rd = m3_cast<double>(mat(FS_AUX + 9));
    m3<double> Sd;
    Sd.a[0][0] = in(FS_AUX + 18);
    Sd.a[0][1] = Sd.a[1][0] = in(FS_AUX + 19);
    Sd.a[0][2] = Sd.a[2][0] = in(FS_AUX + 20);
    Sd.a[1][1] = in(FS_AUX + 21);
    Sd.a[1][2] = Sd.a[2][1] = in(FS_AUX + 22);
    Sd.a[2][2] = in(FS_AUX + 23);
    const double lam = (double)in(FS_CST + KLAM), mu = (double)in(FS_CST + KMU);
    const m3<float> P = m3_cast<float>(pk_from_polar(Fed, Rd, lam, mu));
    const float vol = in(FS_CST + KVOL);
    const float kk = -k3 * a.dt * vol;
    const m3<float> dLdP = kk * mtm(M, Fe);
    const m3<float> dFstress = kk * (M * P);
    const float ax0 = transport();
    const m3<float> Cnext = mat(FS_CNEXT);
    const m3<float> dFn = mat(FS_AF);
    const m3<float> Tr = mtm(m3_eye<float>() + a.dt * Cnext, dFn);
    const m3<float> d2 = m3_cast<float>(d2_mult_from_polar<EXACT, false>(Fed, Rd, Sd, lam, mu, m3_cast<double>(dLdP)));
    m3<float> dLdF, dLdFe;
    if (EXACT) {
        dLdFe = (1.f - a.s) * Tr + dFstress + d2;
        dLdF = dLdFe + a.s * dFn;
    } else {
        dLdF = ((1.f - a.s) * Tr + a.s * dFn) + dFstress + Tr + d2;
        dLdFe = dLdF;
    }
    store_m3(a.adj + (size_t)PF * npl, npl, p, dLdF);
    if (a.ctrl_grad) store_m3(a.ctrl_grad, np, p, dLdFe);
    if (a.ctrl_acc) {
#pragma unroll
        for (int c = 0; c < 3; c++)
#pragma unroll
            for (int r = 0; r < 3; r++)
                a.ctrl_acc[(size_t)(r + 3 * c) * np + p] = in.acc(r + 3 * c) + (double)dLdFe.a[r][c];
    }
    if (a.dbg_dLdP) store_m3(a.dbg_dLdP, np, p, dLdP);
    if (!isfinite(dLdF.a[0][0] + dLdF.a[1][1] + dLdF.a[2][2] + ax0)) atomicOr(a.status, ST_NONFINITE_ADJ);
}

}  // namespace dmpm
