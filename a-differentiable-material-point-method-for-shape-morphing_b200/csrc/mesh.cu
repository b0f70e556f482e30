// mesh.cu -- point cloud of a watertight triangle mesh on the GPU
// (dmpm_mesh_lattice_points, include/dmpm.h): the reference's
// GeometryLoading::GeneratePointCloudFromWatertightTriangleMesh
// (GeometryLoading.cpp:10-83), which keeps the points of the lattice
// min_point + sampling_dx (i, j, k) whose libigl signed distance with the
// winding-number sign is <= 0, i.e. whose winding number w >= 1/2
// (s = 1 - 2 w, S = s |d|; points exactly on the surface are left out here,
// see the header).
//
// One thread per lattice point sums the solid angles of the mesh in FP64 -- a
// triangle's by the formula of Van Oosterom and Strackee (1983),
// tan(Omega / 2) = det / den, det = a.(b x c),
// den = |a||b||c| + (a.b)|c| + (b.c)|a| + (c.a)|b|,
// with a, b, c its vertices relative to the point.
//   The half angles are summed as the product of the complex numbers den + i det,
// with a count of the times it passes the negative real axis: one atan2 per point
// in place of one per triangle, whose FP64 instructions were the kernel's cost.
//   For all but few points the triangles are cut into a tree of patches.  A
// surface's solid angle from a point is that of any surface with the same boundary
// that the point is not between, so a warp with a point in a patch's bounding box
// goes on to its two halves (a leaf is summed triangle by triangle), and any other
// takes the fan over the patch's boundary edges from one of its vertices, which lies
// in the box too (Jacobson, Kavan and Sorkine-Hornung 2013).  A fan has about
// 4 sqrt(triangles) triangles, each with one new vertex.  2.7M points inside 4.4M
// candidates and 1,152 triangles, kernel ms: 29.8 triangle by triangle with an atan2 each, 9.3
// with one level of patches of up to 64, 3.33 with the tree.
//   The kept points are compacted on the GPU in lattice order.  The lattice
// coordinates are formed in float with the reference's two roundings.
//
// dmpm_mesh_jittered_points uses the same inside test for jittered stratified
// sampling (the synthetic scenes' "per_axis^3 points per cell, one uniformly
// jittered point per sub-cell"), with a counter-based jitter so that the points
// depend only on the seed and the sub-cell, not on the launch.
#include <cuda_runtime.h>

#include <algorithm>
#include <array>
#include <climits>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <map>
#include <new>
#include <numeric>
#include <stdexcept>
#include <unordered_map>
#include <utility>
#include <vector>

#include "dmpm.h"
#include "scratch.cuh"
#include "sort.cuh"

namespace {

// triangles of a leaf patch, at most.  Wall ms at 1,152 / 144 / 24,000 triangles: 16: 8.7 /
// 2.3 / 27.1; 24: 7.8 / 2.5 / 24.5; 40: 7.9 / 2.9 / 24.1; 72: 9.2 / 3.0 / 21.8.
constexpr int kPatchTriangles = 40;
// Candidate points from which the tree is built: it costs the host about 1.1 us a
// triangle, the plain sum the GPU that much per triangle for this many points, so the
// line hardly depends on the mesh.  Wall ms of a call, plain / tree, at 30k, 100k and
// 200k candidates: 1,152 triangles 0.76 / 1.04, 1.10 / 1.15, 2.0 / 1.24; 25,600: 14.4 /
// 22.3, 22.5 / 22.8, 41.8 / 23.2; 250,000: 140 / 278, 223 / 278, 413 / 280.
constexpr long long kTreeCandidates = 100000;

// the lattice point min_point + sampling_dx * (i, j, k): a product and a sum, each rounded to float
struct LatticePoints {
    float mn[3], dx;
    __device__ void operator()(int i, int j, int k, double p[3]) const {
        const int id[3] = {i, j, k};
        for (int a = 0; a < 3; a++) p[a] = (double)__fadd_rn(mn[a], __fmul_rn(dx, (float)id[a]));
    }
};

// SplitMix64 (Steele, Lea and Flood 2014): the 64-bit finaliser of a Weyl sequence
__host__ __device__ inline uint64_t splitmix64(uint64_t z) {
    z += 0x9E3779B97F4A7C15ull;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

// one uniformly jittered point per sub-cell (i, j, k) of spacing sdx:
// min + (index + u) * sdx, u = top 24 bits of splitmix64(seed + 3 q + axis) / 2^24,
// q the sub-cell's linear index -- reproducible on any host
struct JitteredPoints {
    float mn[3], sdx;
    int d1, d2;
    uint64_t seed;
    __device__ void operator()(int i, int j, int k, double p[3]) const {
        const int id[3] = {i, j, k};
        const uint64_t q = ((uint64_t)i * d1 + j) * d2 + k;
        for (int a = 0; a < 3; a++) {
            const float u = (float)(splitmix64(seed + 3 * q + a) >> 40) * (1.f / 16777216.f);
            p[a] = (double)__fadd_rn(mn[a], __fmul_rn(__fadd_rn((float)id[a], u), sdx));
        }
    }
};

// One patch, the tree in depth-first order: its bounding box, its boundary fan's
// edges [e0, e1) around apex (far = 0: no fan that costs less than the triangles),
// the patch after its subtree, and a leaf's triangles [t0, t1).
struct Patch {
    float lo[3], hi[3], apex[3];
    int t0, t1, e0, e1, far, skip;
};

struct Vec {
    double x, y, z;
};
__device__ __forceinline__ Vec rel(const float* v, const double p[3]) { return Vec{v[0] - p[0], v[1] - p[1], v[2] - p[2]}; }
__device__ __forceinline__ double dot(const Vec& a, const Vec& b) { return a.x * b.x + a.y * b.y + a.z * b.z; }

// The sum of half solid angles as arg(re + i im) + 2 pi turns, arg in [-pi, pi]
// with atan2's signs at the cut.
struct AngleSum {
    double re = 1.0, im = 0.0;
    int turns = 0;
    // add atan2(det, den)
    __device__ __forceinline__ void add(double det, double den) {
        if (det == 0.0 && den == 0.0) return;  // atan2 gives 0 (or -0)
        const double r = re * den - im * det, i = re * det + im * den;
        const bool up = !signbit(im) && !signbit(det) && signbit(i), down = signbit(im) && signbit(det) && !signbit(i);
        turns += (up ? 1 : 0) - (down ? 1 : 0);
        re = r;
        im = i;
        const double m = fabs(re) + fabs(im);
        if (!(m > 1e-100 && m < 1e100)) {  // rescale; exact, and NaN stays NaN
            const int e = -ilogb(m);
            if (m > 0.0 && m < 1e308) {
                re = scalbn(re, e);
                im = scalbn(im, e);
            }
        }
    }
    __device__ __forceinline__ double value() const { return 2.0 * M_PI * turns + atan2(im, re); }
};

// mask: a bit per point, count: points kept by each block of 256
template <class Points>
__global__ void __launch_bounds__(256) k_mesh_winding(const float* __restrict__ tri, const float* __restrict__ edges,
                                                      const Patch* __restrict__ patches, int np, Points pts, int d0,
                                                      int d1, int d2, uint32_t* __restrict__ mask,
                                                      uint32_t* __restrict__ count) {
    const long long total = (long long)d0 * d1 * d2;
    const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const bool valid = idx < total;
    const long long q = valid ? idx : total - 1;
    const int i = (int)(q / ((long long)d1 * d2)), j = (int)((q / d2) % d1), k = (int)(q % d2);
    double p[3];
    pts(i, j, k, p);
    AngleSum sum;
    for (int n = 0; n < np;) {
        const Patch& P = patches[n];
        bool near = !P.far;
        if (P.far) {
            bool in = true;
#pragma unroll
            for (int a = 0; a < 3; a++) in &= p[a] >= (double)P.lo[a] && p[a] <= (double)P.hi[a];
            near = __any_sync(0xffffffffu, in || !(p[0] == p[0]));
        }
        n = near ? n + 1 : P.skip;  // an inner patch's halves follow it
        if (near) {
            for (int t = P.t0; t < P.t1; t++) {
                const float* v = tri + 9 * (size_t)t;
                const double ax = v[0] - p[0], ay = v[1] - p[1], az = v[2] - p[2];
                const double bx = v[3] - p[0], by = v[4] - p[1], bz = v[5] - p[2];
                const double cx = v[6] - p[0], cy = v[7] - p[1], cz = v[8] - p[2];
                const double la = sqrt(ax * ax + ay * ay + az * az), lb = sqrt(bx * bx + by * by + bz * bz),
                             lc = sqrt(cx * cx + cy * cy + cz * cz);
                const double det = ax * (by * cz - bz * cy) - ay * (bx * cz - bz * cx) + az * (bx * cy - by * cx);
                const double den = la * lb * lc + (ax * bx + ay * by + az * bz) * lc +
                                   (bx * cx + by * cy + bz * cz) * la + (cx * ax + cy * ay + cz * az) * lb;
                sum.add(det, den);
            }
        } else {
            const Vec a = rel(P.apex, p);
            const double la = sqrt(dot(a, a));
            Vec c{0.0, 0.0, 0.0};
            double lc = 0.0, ca = 0.0;
            for (int e = P.e0; e < P.e1; e++) {  // (apex, b, c) with c carried over where the edges chain
                const float* v = edges + 7 * (size_t)e;
                Vec b = c;
                double lb = lc, ab = ca;
                if (v[6] == 0.f) {
                    b = rel(v, p);
                    lb = sqrt(dot(b, b));
                    ab = dot(a, b);
                }
                c = rel(v + 3, p);
                lc = sqrt(dot(c, c));
                ca = dot(c, a);
                const double det = a.x * (b.y * c.z - b.z * c.y) - a.y * (b.x * c.z - b.z * c.x) + a.z * (b.x * c.y - b.y * c.x);
                sum.add(det, la * lb * lc + ab * lc + dot(b, c) * la + ca * lb);
            }
        }
    }
    const bool keep = valid && sum.value() / (2.0 * M_PI) >= 0.5;  // w = sum Omega / (4 pi)
    const unsigned m = __ballot_sync(0xffffffffu, keep);
    if ((threadIdx.x & 31) == 0) mask[idx >> 5] = m;
    const int kept = __syncthreads_count(keep);
    if (threadIdx.x == 0) count[blockIdx.x] = (uint32_t)kept;
}

// the kept points in lattice order: first[b] = points kept by the blocks before b
template <class Points>
__global__ void __launch_bounds__(256) k_mesh_compact(const uint32_t* __restrict__ mask,
                                                      const uint32_t* __restrict__ first, Points pts, int d0, int d1,
                                                      int d2, long long capacity, float* __restrict__ out) {
    const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const uint32_t m = mask[idx >> 5];
    long long o = first[blockIdx.x];
    for (int u = 0; u < w; u++) o += __popc(mask[(idx >> 5) - w + u]);
    o += __popc(m & ((1u << lane) - 1u));
    if (!((m >> lane) & 1u) || o >= capacity) return;
    const int i = (int)(idx / ((long long)d1 * d2)), j = (int)((idx / d2) % d1), k = (int)(idx % d2);
    double p[3];
    pts(i, j, k, p);
    for (int a = 0; a < 3; a++) out[3 * o + a] = (float)p[a];  // a float value: exact
}

// triangles gathered as 9 floats each, indices checked
int gather_triangles(const float* V, int nv, const int* F, int nf, std::vector<float>& tri) {
    tri.resize((size_t)nf * 9);
    for (int f = 0; f < nf; f++)
        for (int c = 0; c < 3; c++) {
            const int v = F[3 * f + c];
            if (v < 0 || v >= nv) return DMPM_ERR_ARG;
            std::memcpy(&tri[(size_t)f * 9 + 3 * c], V + 3 * (size_t)v, 3 * sizeof(float));
        }
    return DMPM_OK;
}

// The triangles in a tree of patches, split at the median centroid of the longest
// axis, and each patch's boundary edges: 7 floats each, the two ends and 1 where the
// first end is the edge before's second (the edges are chained as far as they go).
struct Mesh {
    std::vector<float> tri, edges;
    std::vector<Patch> patches;
};
// all triangles as one leaf
void one_patch(const std::vector<float>& tri, int nf, Mesh& m) {
    m.tri = tri;
    Patch P{};
    P.t1 = nf;
    P.skip = 1;
    m.patches.push_back(P);
}
class PatchTree {
   public:
    PatchTree(const std::vector<float>& tri, int nf, Mesh& m) : tri_(tri), m_(m), order_((size_t)nf), vid_((size_t)nf * 3) {
        // vertices by position, so that unwelded meshes have inner edges too
        auto hash = [](const std::array<float, 3>& x) {
            uint32_t u[3];
            std::memcpy(u, x.data(), sizeof u);
            return (size_t)splitmix64(((uint64_t)u[0] << 32 | u[1]) ^ splitmix64(u[2]));
        };
        std::unordered_map<std::array<float, 3>, int, decltype(hash)> ids((size_t)nf * 2, hash);
        for (size_t v = 0; v < vid_.size(); v++) {
            const float* x = &tri[3 * v];
            if (!(std::isfinite(x[0]) && std::isfinite(x[1]) && std::isfinite(x[2]))) {
                vid_[v] = -1;  // its patches have no fan
                continue;
            }
            const std::array<float, 3> key{x[0] + 0.f, x[1] + 0.f, x[2] + 0.f};  // -0 + 0 = 0
            const auto it = ids.emplace(key, (int)at_.size());
            if (it.second) at_.push_back(x);
            vid_[v] = it.first->second;
        }
        std::iota(order_.begin(), order_.end(), 0);
        Edges net;
        build(0, nf, net);
    }

   private:
    using Edges = std::map<std::pair<int, int>, int>;  // directed edges that no opposite one cancels
    static void add_edge(Edges& net, int u, int v, int times) {
        const auto back = net.find({v, u});
        if (back != net.end()) {
            const int gone = std::min(times, back->second);
            if ((back->second -= gone) == 0) net.erase(back);
            times -= gone;
        }
        if (times > 0) net[{u, v}] += times;
    }
    float centre(int f, int a) const {
        return tri_[9 * (size_t)f + a] + tri_[9 * (size_t)f + 3 + a] + tri_[9 * (size_t)f + 6 + a];
    }
    // the patch of order_[b, e) and its subtree; its boundary into net
    void build(int b, int e, Edges& net) {
        const size_t self = m_.patches.size();
        m_.patches.push_back(Patch{});
        Patch P{};
        for (int a = 0; a < 3; a++) {
            P.lo[a] = INFINITY;
            P.hi[a] = -INFINITY;
        }
        bool finite = true;
        for (int i = b; i < e; i++)
            for (int c = 0; c < 9; c++) {
                const float x = tri_[9 * (size_t)order_[i] + c];
                finite &= std::isfinite(x);
                P.lo[c % 3] = std::min(P.lo[c % 3], x);
                P.hi[c % 3] = std::max(P.hi[c % 3], x);
            }
        P.t0 = P.t1 = (int)(m_.tri.size() / 9);
        if (finite && e - b > kPatchTriangles) {
            int axis = 0;
            for (int a = 1; a < 3; a++)
                if (P.hi[a] - P.lo[a] > P.hi[axis] - P.lo[axis]) axis = a;
            const int mid = b + (e - b) / 2;
            std::nth_element(order_.begin() + b, order_.begin() + mid, order_.begin() + e,
                             [&](int f, int g) { return centre(f, axis) < centre(g, axis); });
            Edges right;
            build(b, mid, net);
            build(mid, e, right);
            for (const auto& n : right) add_edge(net, n.first.first, n.first.second, n.second);
        } else {
            for (int i = b; i < e; i++) {
                const size_t f = (size_t)order_[i];
                m_.tri.insert(m_.tri.end(), tri_.begin() + 9 * f, tri_.begin() + 9 * f + 9);
                for (int c = 0; c < 3 && finite; c++) {
                    const int u = vid_[3 * f + c], v = vid_[3 * f + (c + 1) % 3];
                    if (u != v) add_edge(net, u, v, 1);
                }
            }
            P.t1 = (int)(m_.tri.size() / 9);
        }
        int left = 0;
        for (const auto& n : net) left += n.second;
        // a fan triangle costs about half of one of the patch's
        P.far = finite && left < 2 * (e - b) ? 1 : 0;
        P.e0 = (int)(m_.edges.size() / 7);
        if (P.far && left > 0) fan(net, P);
        P.e1 = (int)(m_.edges.size() / 7);
        P.skip = (int)m_.patches.size();
        m_.patches[self] = P;
    }
    void fan(Edges net, Patch& P) {
        const int apex = net.begin()->first.first;
        std::copy(at_[apex], at_[apex] + 3, P.apex);
        const size_t first = m_.edges.size();
        int prev = -1, last = -1;  // the chain's end, and the last stored edge's
        while (!net.empty()) {
            auto it = prev >= 0 ? net.lower_bound({prev, INT_MIN}) : net.begin();
            if (it == net.end() || (prev >= 0 && it->first.first != prev)) it = net.begin();
            const auto [u, v] = it->first;
            if (--it->second == 0) net.erase(it);
            prev = v;
            if (u == apex || v == apex) continue;  // an edge at the apex spans no triangle
            const bool follows = m_.edges.size() > first && last == u;
            m_.edges.insert(m_.edges.end(), at_[u], at_[u] + 3);
            m_.edges.insert(m_.edges.end(), at_[v], at_[v] + 3);
            m_.edges.push_back(follows ? 1.f : 0.f);
            last = v;
        }
    }

    const std::vector<float>& tri_;
    Mesh& m_;
    std::vector<int> order_, vid_;
    std::vector<const float*> at_;  // a vertex's position
};

// no C++ exception leaves a C entry: host memory that is not to be had is an error code
template <class Fn> int guarded(Fn f) {
    try {
        return f();
    } catch (const std::bad_alloc&) {
        return DMPM_ERR_OOM;
    } catch (const std::length_error&) {
        return DMPM_ERR_OOM;
    }
}

int cuda_failed() {
    cudaGetLastError();
    return DMPM_ERR_CUDA;
}

// the points of the d0 x d1 x d2 generated ones that lie inside, in order: all
// counted, the first `capacity` of them written to out
template <class Points>
int inside_points(const std::vector<float>& tri, int nf, const Points& pts, const int dims[3], float* out,
                  int64_t capacity, int64_t* count) {
    using namespace dmpm;
    const long long total = (long long)dims[0] * dims[1] * dims[2];
    Mesh m;
    if (total < kTreeCandidates) one_patch(tri, nf, m);
    else PatchTree(tri, nf, m);
    const unsigned blocks = (unsigned)((total + 255) / 256);
    const int tiles = (int)((blocks + SCAN_TILE - 1) / SCAN_TILE);
    dmpm_host::Scratch mem;
    float* dtri = mem.alloc<float>(m.tri.size() + m.edges.size());
    Patch* dpat = mem.alloc<Patch>(m.patches.size());
    uint32_t* dmask = mem.alloc<uint32_t>((size_t)blocks * 9 + tiles + 2);
    if (!dtri || !dpat || !dmask) return DMPM_ERR_OOM;
    float* dedge = dtri + m.tri.size();
    uint32_t *dcount = dmask + (size_t)blocks * 8, *dtot = dcount + blocks, *dgrand = dtot + tiles;
    if (cudaMemcpy(dtri, m.tri.data(), m.tri.size() * sizeof(float), cudaMemcpyHostToDevice) != cudaSuccess ||
        (!m.edges.empty() &&
         cudaMemcpy(dedge, m.edges.data(), m.edges.size() * sizeof(float), cudaMemcpyHostToDevice) != cudaSuccess) ||
        cudaMemcpy(dpat, m.patches.data(), m.patches.size() * sizeof(Patch), cudaMemcpyHostToDevice) != cudaSuccess)
        return cuda_failed();
    k_mesh_winding<Points><<<blocks, 256>>>(dtri, dedge, dpat, (int)m.patches.size(), pts, dims[0], dims[1], dims[2],
                                            dmask, dcount);
    k_scan_tiles<OpSum><<<tiles, SCAN_THREADS>>>(dcount, (int)blocks, dtot);
    k_scan_totals<OpSum><<<1, 1024>>>(dtot, tiles, dgrand);
    k_scan_add<OpSum><<<tiles, SCAN_THREADS>>>(dcount, (int)blocks, dtot);
    uint32_t n = 0;
    if (cudaGetLastError() != cudaSuccess || cudaMemcpy(&n, dgrand, 4, cudaMemcpyDeviceToHost) != cudaSuccess)
        return cuda_failed();
    *count = n;
    const int64_t write = std::min<int64_t>(n, capacity);
    if (write > 0) {
        float* dout = mem.alloc<float>((size_t)write * 3);
        if (!dout) return DMPM_ERR_OOM;
        k_mesh_compact<Points><<<blocks, 256>>>(dmask, dcount, pts, dims[0], dims[1], dims[2], write, dout);
        if (cudaGetLastError() != cudaSuccess ||
            cudaMemcpy(out, dout, (size_t)write * 12, cudaMemcpyDeviceToHost) != cudaSuccess)
            return cuda_failed();
    }
    return (int64_t)n > capacity ? DMPM_ERR_TOO_LARGE : DMPM_OK;
}

}  // namespace

extern "C" int dmpm_mesh_lattice_dims(const float* min_point, const float* max_point, float sampling_dx, int* dims) {
    if (!min_point || !max_point || !dims || !(sampling_dx > 0.f)) return DMPM_ERR_ARG;
    for (int a = 0; a < 3; a++) {
        const float ext = max_point[a] - min_point[a];
        const double d = std::ceil((double)(ext / sampling_dx)) + 1.0;  // GeometryLoading.cpp:21-23
        if (!(d >= 1.0) || d > 1e6) return DMPM_ERR_ARG;
        dims[a] = (int)d;
    }
    return DMPM_OK;
}

extern "C" int dmpm_mesh_lattice_points(const float* V, int nv, const int* F, int nf, const float* min_point,
                                        const float* max_point, float sampling_dx, float* out, int64_t capacity,
                                        int64_t* count) {
    if (!V || nv < 3 || !F || nf < 1 || !count || capacity < 0 || (capacity > 0 && !out)) return DMPM_ERR_ARG;
    int dims[3];
    int st = dmpm_mesh_lattice_dims(min_point, max_point, sampling_dx, dims);
    if (st != DMPM_OK) return st;
    const long long total = (long long)dims[0] * dims[1] * dims[2];
    if (total > (1ll << 31)) return DMPM_ERR_TOO_LARGE;
    const LatticePoints pts{{min_point[0], min_point[1], min_point[2]}, sampling_dx};
    return guarded([&] {
        std::vector<float> tri;
        const int bad = gather_triangles(V, nv, F, nf, tri);
        return bad != DMPM_OK ? bad : inside_points(tri, nf, pts, dims, out, capacity, count);
    });
}

extern "C" int dmpm_mesh_jittered_points(const float* V, int nv, const int* F, int nf, const float* min_point,
                                         const float* max_point, float cell_dx, int per_axis, uint64_t seed,
                                         float* out, int64_t capacity, int64_t* count) {
    if (!V || nv < 3 || !F || nf < 1 || !count || capacity < 0 || (capacity > 0 && !out) || !min_point ||
        !max_point || !(cell_dx > 0.f) || per_axis < 1 || per_axis > 64)
        return DMPM_ERR_ARG;
    int dims[3];
    for (int a = 0; a < 3; a++) {
        const double c = std::ceil((double)((max_point[a] - min_point[a]) / cell_dx));
        if (!(c >= 1.0) || c * per_axis > 1e6) return DMPM_ERR_ARG;
        dims[a] = (int)c * per_axis;
    }
    const long long total = (long long)dims[0] * dims[1] * dims[2];
    if (total > (1ll << 31)) return DMPM_ERR_TOO_LARGE;
    const float sdx = cell_dx / (float)per_axis;
    const JitteredPoints pts{{min_point[0], min_point[1], min_point[2]}, sdx, dims[1], dims[2], seed};
    return guarded([&] {
        std::vector<float> tri;
        const int bad = gather_triangles(V, nv, F, nf, tri);
        return bad != DMPM_OK ? bad : inside_points(tri, nf, pts, dims, out, capacity, count);
    });
}
