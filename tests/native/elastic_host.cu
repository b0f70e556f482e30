// elastic_host.cu -- the two forms of the reference-style stress derivative
// (csrc/elasticity.cuh: d2_mult_from_polar<false, FD>) for the host, for
// tests/test_elastic_host.py.  Test infrastructure only.
#include "elasticity.cuh"

using namespace dmpm;

static m3<double> ld(const double* a) {  // row-major
    m3<double> m;
    for (int i = 0; i < 3; i++) for (int j = 0; j < 3; j++) m.a[i][j] = a[3 * i + j];
    return m;
}
extern "C" void eh_d2(const double* F, const double* R, const double* S, double lam, double mu, const double* dF, int fd,
                      double* out) {
    const m3<double> d = fd ? d2_mult_from_polar<false, true>(ld(F), ld(R), ld(S), lam, mu, ld(dF))
                            : d2_mult_from_polar<false, false>(ld(F), ld(R), ld(S), lam, mu, ld(dF));
    for (int i = 0; i < 3; i++) for (int j = 0; j < 3; j++) out[3 * i + j] = d.a[i][j];
}
