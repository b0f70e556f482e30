"""The FP32 path's kernels over chunks of 32 sorted particles, at the sizes where
a chunk, a block or a group of equal stencil bases ends: clouds of 1 to a few
hundred particles on a non-cubic grid, some of them at and outside its faces,
moving up to a cell between sorts so that chunks hold particles that have left
their cells.  The FP64 oracle is the CPU restatement of the reference's
ForwardTimeStep / EndLayerMassLoss / Back_Timestep; node sums add up to a few
hundred float terms (a few times 1e-6 of their size), and the bars are those of
the other FP32 tests."""
import numpy as np
import pytest

import scenes
from oracle.lib import OracleGraph
from tests.helpers import normrel, relerr
from tests.test_gpu_parity import make_ctx

pytestmark = pytest.mark.gpu

L = 5


def _cloud(n, seed):
    rng = np.random.default_rng(seed)
    dims = (9, 7, 11)
    x = rng.uniform(0.0, 1.0, (n, 3)) * (np.array(dims) - 1.0)
    if n > 8:
        x[::8] = np.array(dims) - 1.0 + rng.uniform(-0.4, 0.4, (len(x[::8]), 3))  # at the far corner, some outside
        x[1::16] = x[2]  # a crowd in one cell
        x[1::16] += rng.uniform(-0.05, 0.05, (len(x[1::16]), 3))
    z = np.zeros((n, 3, 3))
    sc = scenes.Scene(name="cloud", x=x, v=rng.normal(0.0, 3.0, (n, 3)), F=z + np.eye(3), C=rng.normal(0, 0.1, (n, 3, 3)),
                      dFc=rng.normal(0.0, 1e-3, (n, 3, 3)), m=rng.uniform(0.5, 2.0, n), lam=np.full(n, 50.0),
                      mu=np.full(n, 40.0), vol=np.full(n, 0.3), dims=dims, dx=1.0, min_point=np.zeros(3),
                      target_points=rng.uniform(2.0, 5.0, (50, 3)), target_mp=1.0, dt=0.05, steps=L - 1, drag=0.2,
                      smoothing=0.1, f_ext=np.array([0.0, -1.0, 0.5]))
    return sc.float32_inputs()


@pytest.mark.parametrize("n,general,adjoint", [(1, False, "exact"), (2, False, "refcompat"), (31, False, "exact"),
                                               (32, True, "exact"), (33, False, "exact"), (33, False, "refcompat"),
                                               (127, False, "exact"), (128, False, "exact"), (129, True, "refcompat"),
                                               (129, False, "exact"), (421, False, "refcompat"), (421, False, "exact")])
def test_chunks_match_fp64_oracle(gpu_ready, n, general, adjoint):
    sc = _cloud(n, 100 + n)
    o = OracleGraph(sc, "f64")
    o.setup(L, sc.dt, sc.drag, sc.f_ext, sc.smoothing)
    o.forward(0)
    loss = o.loss()
    o.backward(0, 1 if adjoint == "exact" else 0)
    with make_ctx(sc, "fp32", o.target, adjoint=adjoint, keep_adjoints=True, sort_every=50, warp_general=general) as c:
        c.setup(L)
        c.forward(0)
        assert abs(c.loss() - loss) <= 1e-4 * abs(loss)
        c.backward(0)
        for l in (0, L - 2):
            assert relerr(c.get_grid(l, "grid_m"), o.get(l, "grid_m")) < 1e-5
            assert relerr(c.get_grid(l, "grid_p"), o.get(l, "grid_p")) < 2e-4
        for f, bar in (("x", 1e-5), ("F", 1e-4), ("v", 2e-3), ("C", 2e-3)):
            assert relerr(c.get(L - 1, f), o.get(L - 1, f)) < bar, f
        for f in ("dLdx", "dLdv", "dLdF", "dLdC", "dLdFe"):
            if f == "dLdFe" and adjoint != "exact":
                continue
            assert normrel(c.get(0, f), o.get(0, f)) < 1e-3, f


@pytest.mark.parametrize("n,adjoint", [(1, "exact"), (31, "exact"), (33, "refcompat"), (128, "exact"), (129, "exact"),
                                       (421, "refcompat"), (421, "exact")])
def test_fp64_chunks_match_fp64_oracle(gpu_ready, n, adjoint):
    """The FP64 path's P2G and adjoint scatter over chunks: the bars of the other
    FP64 tests, as the sums differ from the oracle's by their order alone."""
    sc = _cloud(n, 300 + n)
    o = OracleGraph(sc, "f64")
    o.setup(L, sc.dt, sc.drag, sc.f_ext, sc.smoothing)
    o.forward(0)
    loss = o.loss()
    o.backward(0, 1 if adjoint == "exact" else 0)
    with make_ctx(sc, "fp64", o.target, adjoint=adjoint, keep_adjoints=True, sort_every=50) as c:
        c.setup(L)
        c.forward(0)
        assert abs(c.loss() - loss) <= 1e-10 * abs(loss)
        c.backward(0)
        for l in (0, L - 2):
            assert relerr(c.get_grid(l, "grid_m"), o.get(l, "grid_m")) < 1e-10
            assert relerr(c.get_grid(l, "grid_p"), o.get(l, "grid_p")) < 1e-10
        for f in ("x", "F", "v", "C"):
            assert relerr(c.get(L - 1, f), o.get(L - 1, f)) < 1e-10, f
        for f in ("dLdx", "dLdv", "dLdF", "dLdC"):
            assert normrel(c.get(0, f), o.get(0, f)) < 1e-8, f
