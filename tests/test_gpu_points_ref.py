"""dmpm_get_points_ref on clouds that end with or just after one of its pinned buffers
(2,148 points with adjoints, 3,542 without) and on larger ones, whose rows several host
threads write (above 34,379 and 56,680 points): every field the engine fills equals what
dmpm_get_particles returns, rounded to float, in the caller's order, and the other floats
of the structs stay as they were."""
import numpy as np
import pytest

import scenes
from tests.test_gpu_parity import make_ctx

pytestmark = pytest.mark.gpu

# field, first float in the struct
STATE = (("x", 0), ("v", 3), ("F", 6), ("C", 15), ("m", 33), ("vol", 34), ("lam", 35), ("mu", 36), ("dFc", 37))
ADJOINT = (("dLdx", 46), ("dLdv", 49), ("dLdF", 52), ("dLdC", 61))


@pytest.mark.parametrize("n", [1, 2148, 2149, 3542, 3543, 40013, 70001])
@pytest.mark.parametrize("prec,reorder", [("fp32", False), ("fp32", True), ("fp64", False)])
def test_every_row_of_every_buffer(gpu_ready, n, prec, reorder):
    rng = np.random.default_rng(n)
    dims = (24, 20, 22)
    x = rng.uniform(3.0, 17.0, (n, 3))
    sc = scenes.Scene(name="cloud", x=x, v=rng.normal(0.0, 1.0, (n, 3)), F=np.eye(3) + rng.normal(0, 0.01, (n, 3, 3)),
                      C=rng.normal(0, 0.1, (n, 3, 3)), dFc=rng.normal(0.0, 1e-3, (n, 3, 3)), m=rng.uniform(0.5, 2.0, n),
                      lam=rng.uniform(40.0, 60.0, n), mu=rng.uniform(30.0, 50.0, n), vol=rng.uniform(0.2, 0.4, n),
                      dims=dims, dx=1.0, min_point=np.zeros(3), target_points=x[:50], target_mp=1.0, dt=0.01, steps=2,
                      drag=0.0, smoothing=0.0, f_ext=np.zeros(3)).float32_inputs()
    with make_ctx(sc, prec, rng.uniform(0.0, 2.0, int(np.prod(dims))), adjoint="exact", reorder_particles=reorder) as c:
        c.setup(3)
        c.forward(0)
        for layer, adjoints in ((1, False), (2, True), (0, True)):
            if layer == 2:
                c.loss()
            if layer == 0:
                c.backward(0)
            mark = rng.normal(0.0, 1.0, (n, 118)).astype(np.float32)
            out = c.get_points_ref(layer, mark.copy())
            filled = np.zeros(118, dtype=bool)
            for f, at in STATE + (ADJOINT if adjoints else ()):
                a = c.get(layer, f)
                a = (a.transpose(0, 2, 1) if a.ndim == 3 else a).reshape(n, -1).astype(np.float32)
                assert np.array_equal(out[:, at:at + a.shape[1]], a), (layer, f)
                filled[at:at + a.shape[1]] = True
            assert np.array_equal(out[:, ~filled], mark[:, ~filled])
