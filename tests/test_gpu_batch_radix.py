"""A batch whose grids together have more than 4M cell keys and 32 per particle, so that
its cell order comes from the radix sort, against one engine context per instance (which
sorts the same way).  Both sum in float, in another order; the bars are those of the
batch's other tests."""
import numpy as np
import pytest

import dmpm
import scenes
from oracle.lib import OracleGraph  # noqa: F401
from tests.helpers import normrel, relerr
from tests.test_gpu_parity import make_ctx

pytestmark = pytest.mark.gpu


def _scene(seed, dims, n, steps):
    rng = np.random.default_rng(seed)
    x = np.array(dims) / 2.0 + rng.uniform(-4.0, 4.0, (n, 3))
    return scenes.Scene(name="cloud", x=x, v=rng.normal(0.0, 1.0, (n, 3)) + np.array([4.0, 0.0, 0.0]),
                        F=np.zeros((n, 3, 3)) + np.eye(3), C=rng.normal(0, 0.1, (n, 3, 3)),
                        dFc=rng.normal(0.0, 1e-3, (n, 3, 3)), m=rng.uniform(0.5, 2.0, n), lam=np.full(n, 50.0),
                        mu=np.full(n, 40.0), vol=np.full(n, 0.3), dims=dims, dx=1.0, min_point=np.zeros(3),
                        target_points=x[:50], target_mp=1.0, dt=0.05, steps=steps, drag=0.2, smoothing=0.1,
                        f_ext=np.array([0.0, -1.0, 0.5])).float32_inputs()


@pytest.mark.parametrize("graph", [False, True])
def test_batch_over_the_radix_sort(gpu_ready, graph):
    scs = [_scene(1, (260, 260, 60), 1500, 4), _scene(2, (24, 20, 22), 700, 6), _scene(3, (90, 260, 60), 33, 2)]
    targets = [np.random.default_rng(9 + i).uniform(0.0, 2.0, int(np.prod(s.dims))) for i, s in enumerate(scs)]
    with dmpm.Batch([{"n": s.n, "dims": s.dims, "dx": s.dx, "min_point": s.min_point, "steps": s.steps} for s in scs]) as b:
        b.set_params(scs[0].dt, drag=0.2, smoothing=0.1, f_ext=scs[0].f_ext, adjoint="exact")
        for i, s in enumerate(scs):
            b.set_particles(i, s.x, s.m, s.lam, s.mu, v=s.v, F=s.F, C=s.C, dFc=s.dFc, vol=s.vol)
            b.set_target_mass(i, targets[i])
        b.set_launch(sort_every=3, use_graph=graph)
        b.setup()
        for _ in range(2):
            losses = b.gradient()
            for i, s in enumerate(scs):
                with make_ctx(s, "fp32", targets[i], adjoint="exact", control="tied", sort_every=3) as c:
                    c.setup(s.steps + 1)
                    c.forward(0)
                    assert abs(losses[i] - c.loss()) <= 1e-5 * abs(losses[i]), i
                    c.backward(0)
                    assert relerr(b.get(i, s.steps, "x"), c.get(s.steps, "x")) < 1e-5, i
                    assert normrel(b.control_grad(i), c.control_grad()) < 1e-3, i


def test_fp64_path_over_the_radix_sort(gpu_ready):
    """The FP64 path on a grid whose order comes from the radix sort against the same cloud, moved by
    whole cells, on one that counts: the same sums in another order, positions to the rounding of
    coordinates of 130 cells (an absolute 3e-14, amplified by the node masses' quotients)."""
    a = _scene(1, (260, 260, 60), 1500, 3)
    b = _scene(1, (260, 260, 60), 1500, 3)
    shift = np.array([98.0, 115.0, 15.0])
    b.x = a.x - shift  # exact: float32 positions below 256 less whole numbers
    b.dims = (64, 30, 30)
    out = []
    for s in (a, b):
        with make_ctx(s, "fp64", np.zeros(int(np.prod(s.dims))), adjoint="exact", control="tied", sort_every=2) as c:
            c.setup(s.steps + 1)
            c.forward(0)
            c.loss()
            c.backward(0)
            out.append((c.get(s.steps, "x"), c.get(s.steps, "F"), c.control_grad()))
    assert np.abs(out[0][0] - shift - out[1][0]).max() < 1e-10
    assert relerr(out[0][1], out[1][1]) < 1e-10
    assert normrel(out[0][2], out[1][2]) < 1e-8
