"""Node boxes of the FP32 path: the node passes walk each layer's box of touched
nodes, so a grid that is used again must be cleared over its old box before the
box takes in where the cloud has got to.  The cloud here is sparse, spans more
rows of nodes than a node pass has warps (about 115 x 115 against 9,472), and
expands by about a cell per step, so boxes that hold an earlier pass's nodes grow
at every step.  The deterministic mode in a context of its own is the oracle: it
runs its node passes over whole grids, in the same arithmetic.  Node sums add a
few tens of float terms (relative rounding 1e-6 of the largest), while a node left
uncleared is wrong by its whole mass; the bars are those of the other FP32 tests."""
import numpy as np
import pytest

import scenes
from tests.helpers import normrel, relerr
from tests.test_gpu_parity import make_ctx

pytestmark = pytest.mark.gpu

L = 7
DIMS = (128, 128, 16)


def _sparse(seed, lo=8.0, cells=28, alpha=0.2):
    """cells^2 particles, 4 cells apart on the first two axes, in the expanding motion
    v = alpha (x - centre): 1.1 cells per step at the rim of 28^2"""
    rng = np.random.default_rng(seed)
    i, j = np.meshgrid(np.arange(cells), np.arange(cells), indexing="ij")
    n = i.size
    x = np.stack([lo + 4.0 * i.ravel(), lo + 4.0 * j.ravel(), rng.uniform(5.0, 10.0, n)], axis=1)
    x[:, :2] += rng.uniform(0.0, 2.0, (n, 2))
    centre = x[:, :2].mean(axis=0)
    v = np.zeros((n, 3))
    v[:, :2] = alpha * (x[:, :2] - centre)
    C = np.zeros((n, 3, 3))
    C[:, 0, 0] = C[:, 1, 1] = alpha
    sc = scenes.Scene(name="sparse", x=x, v=v, F=np.zeros((n, 3, 3)) + np.eye(3), C=C,
                      dFc=rng.normal(0.0, 1e-3, (n, 3, 3)), m=rng.uniform(0.5, 2.0, n), lam=np.full(n, 2.0),
                      mu=np.full(n, 1.5), vol=np.full(n, 0.3), dims=DIMS, dx=1.0, min_point=np.zeros(3),
                      target_points=rng.uniform(20.0, 100.0, (50, 3)), target_mp=1.0, dt=0.1, steps=L - 1, drag=0.0,
                      smoothing=0.0, f_ext=np.zeros(3))
    return sc.float32_inputs()


def _target(seed):
    return np.random.default_rng(seed).uniform(0.0, 0.2, int(np.prod(DIMS)))


def _gradient(c):
    c.forward(0)
    loss = c.loss()
    c.backward(0)
    return loss


def _check(c, sc, ref):
    """c after _gradient against ref, a context that has run the same in the other mode"""
    for l in range(L - 1):
        m = c.get_grid(l, "grid_m")
        assert abs(m.sum() - sc.m.sum()) <= 1e-5 * sc.m.sum(), l
        assert relerr(m, ref.get_grid(l, "grid_m")) < 1e-5, l
        assert relerr(c.get_grid(l, "grid_p"), ref.get_grid(l, "grid_p")) < 2e-4, l
    assert relerr(c.get(L - 1, "x"), ref.get(L - 1, "x")) < 1e-5
    assert relerr(c.get(L - 1, "F"), ref.get(L - 1, "F")) < 1e-4
    for f in ("dLdx", "dLdv", "dLdF", "dLdC"):
        assert normrel(c.get(0, f), ref.get(0, f)) < 1e-3, f


def _reference(sc, target, **kw):
    ref = make_ctx(sc, "fp32", target, adjoint="exact", deterministic=True, **kw)
    ref.setup(L)
    return ref, _gradient(ref)


@pytest.mark.parametrize("checkpoint", [2, 3, L])
def test_checkpointed_grids_are_cleared(gpu_ready, checkpoint):
    sc, target = _sparse(1), _target(2)
    ref, loss = _reference(sc, target)
    with ref, make_ctx(sc, "fp32", target, adjoint="exact", checkpoint_every=checkpoint) as c:
        c.setup(L)
        for _ in range(2):  # the second pass begins with the first one's grids
            assert abs(_gradient(c) - loss) <= 1e-4 * abs(loss)
            _check(c, sc, ref)


@pytest.mark.parametrize("eager", [False, True])
def test_second_evaluation_with_wider_motion(gpu_ready, eager):
    slow, wide, target = _sparse(1, alpha=0.05), _sparse(1), _target(2)
    ref, loss = _reference(wide, target, checkpoint_every=1)
    with ref, make_ctx(slow, "fp32", target, adjoint="exact", checkpoint_every=1, eager=eager) as c:
        c.setup(L)
        _gradient(c)
        for f, a in (("v", wide.v), ("C", wide.C)):
            c.set_layer(0, f, a)
        assert abs(_gradient(c) - loss) <= 1e-4 * abs(loss)
        _check(c, wide, ref)


@pytest.mark.parametrize("checkpoint", [1, 3])
def test_positions_set_between_passes(gpu_ready, checkpoint):
    """Positions of a layer set after the forward pass: the adjoint's stencils then lie outside the
    box that the layer's P2G left.  The next forward pass overwrites them."""
    sc, target = _sparse(1), _target(2)
    kw = dict(adjoint="exact", checkpoint_every=checkpoint)

    def run(c):
        out = []
        c.setup(L)
        _gradient(c)
        x3 = c.get(3, "x")
        for edit in (np.array([0.0, 0.0, -4.0]), np.array([-6.0, 5.0, 4.5])):
            c.set_layer(3, "x", x3 + edit)
            c.loss()
            c.backward(0)
            out.append([c.get(0, f) for f in ("dLdx", "dLdv", "dLdF", "dLdC")])
        _gradient(c)
        out.append([c.get(0, f) for f in ("dLdx", "dLdv", "dLdF", "dLdC")])
        return out

    with make_ctx(sc, "fp32", target, deterministic=True, **kw) as ref, make_ctx(sc, "fp32", target, **kw) as c:
        want, got = run(ref), run(c)
    for i, (w, g) in enumerate(zip(want, got)):
        for a, b in zip(w, g):
            assert normrel(b, a) < 1e-3, i


@pytest.mark.parametrize("checkpoint", [1, 2])
def test_float_passes_after_deterministic_ones_and_a_second_cloud(gpu_ready, checkpoint):
    """Deterministic passes leave whole grids of nodes, a second cloud of the same size starts elsewhere."""
    a, b, target = _sparse(1, cells=20), _sparse(4, lo=40.0, cells=20), _target(2)
    kw = dict(adjoint="exact", checkpoint_every=checkpoint)

    def params(c, sc, deterministic):
        c.set_params(dt=sc.dt, drag=sc.drag, f_ext=sc.f_ext, smoothing=sc.smoothing, deterministic=deterministic, **kw)

    with make_ctx(a, "fp32", target, **kw) as c:
        c.setup(L)
        for sc in (a, b, a):
            c.set_particles(sc.x, sc.m, sc.lam, sc.mu, v=sc.v, F=sc.F, C=sc.C, dFc=sc.dFc, vol=sc.vol)
            c.setup(L)
            ref, loss = _reference(sc, target)
            with ref:
                for deterministic in (False, True, False, False):
                    params(c, sc, deterministic)
                    assert abs(_gradient(c) - loss) <= 1e-4 * abs(loss)
                    _check(c, sc, ref)
