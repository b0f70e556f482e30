"""The deterministic mode set and taken back between the passes of one context
(FP32 path).  Its P2G and adjoint scatter read warp items, which the float mode's
sorts do not form -- neither the counting sort nor, on grids of more than 32 cell
keys per particle and 4M keys, the radix sort -- so a pass must sort again for
them; and each mode's node passes must leave sums, boxes and adjoint grids as the
other expects them.  The oracle is a context that stays in the deterministic mode;
both modes compute the same quantities in float, so the bars are those between
the FP32 path and its oracle elsewhere."""
import numpy as np
import pytest

import scenes
from tests.helpers import normrel, relerr
from tests.test_gpu_parity import make_ctx

pytestmark = pytest.mark.gpu

L = 6


def _scene(dims, n=1500):
    """a drifting, stirred cloud of 8^3 cells in the middle of the grid"""
    rng = np.random.default_rng(5)
    x = np.array(dims) / 2.0 + rng.uniform(-4.0, 4.0, (n, 3))
    sc = scenes.Scene(name="cloud", x=x, v=rng.normal(0.0, 1.0, (n, 3)) + np.array([4.0, 0.0, 0.0]),
                      F=np.zeros((n, 3, 3)) + np.eye(3), C=rng.normal(0, 0.1, (n, 3, 3)),
                      dFc=rng.normal(0.0, 1e-3, (n, 3, 3)), m=rng.uniform(0.5, 2.0, n), lam=np.full(n, 50.0),
                      mu=np.full(n, 40.0), vol=np.full(n, 0.3), dims=dims, dx=1.0, min_point=np.zeros(3),
                      target_points=x[:50] + 3.0, target_mp=1.0, dt=0.05, steps=L - 1, drag=0.2, smoothing=0.1,
                      f_ext=np.array([0.0, -1.0, 0.5]))
    return sc.float32_inputs()


# 64 x 30 x 30 nodes: counting sort; 260 x 260 x 60: 4.7M cell keys, radix sort
@pytest.mark.parametrize("dims", [(64, 30, 30), (260, 260, 60)])
@pytest.mark.parametrize("checkpoint", [1, 2])
@pytest.mark.parametrize("eager", [False, True])
def test_modes_switched_between_passes(gpu_ready, dims, checkpoint, eager):
    sc = _scene(dims)
    target = np.zeros(int(np.prod(dims)))
    kw = dict(adjoint="exact", control="tied", checkpoint_every=checkpoint, eager=eager, sort_every=4)

    def mode(c, deterministic):
        c.set_params(dt=sc.dt, drag=sc.drag, f_ext=sc.f_ext, smoothing=sc.smoothing, deterministic=deterministic, **kw)

    with make_ctx(sc, "fp32", target, deterministic=True, **kw) as c:
        c.setup(L)
        c.forward(0)
        loss = c.loss()
        c.backward(0)
        grad, dldx, x = c.control_grad(), c.get(0, "dLdx"), c.get(L - 1, "x")

    def check(c, what):
        assert abs(c.loss() - loss) <= 1e-4 * abs(loss), what
        c.backward(0)
        assert relerr(c.get(L - 1, "x"), x) < 1e-5, what
        assert normrel(c.control_grad(), grad) < 1e-3, what
        assert normrel(c.get(0, "dLdx"), dldx) < 1e-3, what

    with make_ctx(sc, "fp32", target, **kw) as c:
        c.setup(L)
        c.forward(0)
        check(c, "float")
        mode(c, True)
        check(c, "float states, deterministic adjoint")
        c.forward(2)  # within the first sort interval
        check(c, "deterministic from layer 2")
        mode(c, False)
        check(c, "back to float")
        c.forward(0)
        check(c, "float again")
        mode(c, True)
        c.forward(0)
        check(c, "deterministic")
        mode(c, False)
        c.forward(0)
        check(c, "float after it")
        c.set_particles(sc.x, sc.m, sc.lam, sc.mu, v=sc.v, F=sc.F, C=sc.C, dFc=sc.dFc, vol=sc.vol)
        mode(c, True)
        c.setup(L)
        c.forward(0)
        assert c.loss() == loss
        c.backward(0)
        assert np.array_equal(c.control_grad(), grad)
