"""The chunk kernels on either side of the cloud sizes at which their launches change:
8, 16 or 32 sorted particles per warp of the scatters (from 18,944 and 37,888 particles,
in the FP64 path from 5,920 and 11,840), four threads or one per particle in G2P and the
adjoint gather (from 14,500), with ragged last warps and blocks.  tests/test_gpu_chunk.py
has the small sizes, all of which run 8 per warp and four threads per particle.  The
oracle is the CPU restatement of the reference in FP64; about 5 particles per cell and a
crowd of some hundred in one, so node sums add a few hundred to a thousand float terms,
and the bars are those of that file."""
import numpy as np
import pytest

import scenes
from oracle.lib import OracleGraph
from tests.helpers import normrel, relerr
from tests.test_gpu_parity import make_ctx

pytestmark = pytest.mark.gpu

L = 4


def _cloud(n, seed):
    rng = np.random.default_rng(seed)
    dims = (20, 17, 23)
    x = rng.uniform(0.0, 1.0, (n, 3)) * (np.array(dims) - 1.0)
    x[:300] = np.array(dims) / 2.0 + rng.uniform(-0.3, 0.3, (300, 3))  # a crowd
    x[300:400] = np.array(dims) - 1.0 + rng.uniform(-0.4, 0.4, (100, 3))  # at the far corner, some outside
    x = x[rng.permutation(n)]
    sc = scenes.Scene(name="cloud", x=x, v=rng.normal(0.0, 3.0, (n, 3)), F=np.zeros((n, 3, 3)) + np.eye(3),
                      C=rng.normal(0, 0.1, (n, 3, 3)), dFc=rng.normal(0.0, 1e-3, (n, 3, 3)), m=rng.uniform(0.5, 2.0, n),
                      lam=np.full(n, 50.0), mu=np.full(n, 40.0), vol=np.full(n, 0.3), dims=dims, dx=1.0,
                      min_point=np.zeros(3), target_points=rng.uniform(2.0, 12.0, (500, 3)), target_mp=1.0, dt=0.05,
                      steps=L - 1, drag=0.2, smoothing=0.1, f_ext=np.array([0.0, -1.0, 0.5]))
    return sc.float32_inputs()


@pytest.fixture(scope="module", params=[5919, 5921, 11839, 11841, 14499, 14500, 18943, 18945, 37887, 37889, 39999, 40001, 41107])
def cloud(request):
    sc = _cloud(request.param, request.param)
    exact = request.param % 4 != 1  # both adjoints over the list
    o = OracleGraph(sc, "f64")
    o.setup(L, sc.dt, sc.drag, sc.f_ext, sc.smoothing)
    o.forward(0)
    loss = o.loss()
    o.backward(0, 1 if exact else 0)
    return sc, o, loss, "exact" if exact else "refcompat"


def test_fp32_matches_fp64_oracle(gpu_ready, cloud):
    sc, o, loss, adjoint = cloud
    with make_ctx(sc, "fp32", o.target, adjoint=adjoint, keep_adjoints=True, sort_every=50) as c:
        c.setup(L)
        c.forward(0)
        assert abs(c.loss() - loss) <= 1e-4 * abs(loss)
        c.backward(0)
        for l in (0, L - 2):
            assert relerr(c.get_grid(l, "grid_m"), o.get(l, "grid_m")) < 1e-5
            assert relerr(c.get_grid(l, "grid_p"), o.get(l, "grid_p")) < 2e-4
        for f, bar in (("x", 1e-5), ("F", 1e-4), ("v", 2e-3), ("C", 2e-3)):
            assert relerr(c.get(L - 1, f), o.get(L - 1, f)) < bar, f
        for f in ("dLdx", "dLdv", "dLdF", "dLdC"):
            assert normrel(c.get(0, f), o.get(0, f)) < 1e-3, f


def test_fp64_matches_fp64_oracle(gpu_ready, cloud):
    sc, o, loss, adjoint = cloud
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
