// nodes_host.cu -- the node addressing of the FP32 gathers (StencilNodes,
// csrc/kernels_chunk.cuh) for the host, for tests/test_nodes_host.py.
// Test infrastructure only.
#include "kernels_chunk.cuh"

using namespace dmpm;

// record index of node (base + (i, j, 0)), R records per node
template <bool INSIDE, int R> static long long record(const int* dim, int goff, const int* base, int i, int j) {
    GridGeom g{};
    for (int c = 0; c < 3; c++) g.dim[c] = dim[c];
    // an address with room on both sides; nothing is read
    const uintptr_t zero = (uintptr_t)1 << 46;
    const StencilNodes<INSIDE, R> n((const node4<float>*)zero, g, goff, base);
    return ((long long)(uintptr_t)n.row(i, j) - (long long)zero) / (long long)sizeof(node4<float>);
}
extern "C" long long nh_record(const int* dim, int goff, const int* base, int i, int j, int pair, int inside) {
    if (pair) return inside ? record<true, 2>(dim, goff, base, i, j) : record<false, 2>(dim, goff, base, i, j);
    return inside ? record<true, 1>(dim, goff, base, i, j) : record<false, 1>(dim, goff, base, i, j);
}
