"""bench.py's bytes per launch, from which its bandwidth fractions are formed: the
float mode's kernels as they run, and nothing for the deterministic mode, whose
kernels it does not describe (integer sums over the whole grid, the stress stage and
the adjoint's sources in kernels of their own)."""
import os
import sys

import pytest

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, REPO)
import bench  # noqa: E402


# bytes per particle and touched node of a launch
KERNELS = {"p_op1": (220, 0), "p2g": (80, 16), "g_op": (0, 48), "g2p_p_op2": (356, 16), "adj_g2p_scatter": (244, 16),
           "adj_g_op": (0, 80), "adj_p2g_gather": (596, 32), "p2g_mass": (28, 4), "loss_dldx": (124, 4)}


@pytest.mark.parametrize("kernel", KERNELS)
def test_bytes_of_the_float_mode(kernel):
    p, t = KERNELS[kernel]
    assert bench.launch_bytes(kernel, 1000, 10) == 1000 * p + 10 * t
    assert bench.launch_bytes(kernel, 1000, 10, deterministic=False) == 1000 * p + 10 * t


def test_kernels_without_a_figure():
    assert bench.launch_bytes("node_loss", 1000, 10) == 0
    for k in KERNELS:
        assert bench.launch_bytes(k, 1000, 10, deterministic=True) == 0


def test_roofline_entry():
    stats = {"adj_p2g_gather": (20.0, 200), "g_op": (1.5, 200)}
    kern, roof = bench.roofline(stats, 1000, 10, 5000.0, "measured", deterministic=False)
    b = 1000 * 596 + 10 * 32
    assert roof["kernel"] == "adj_p2g_gather" and roof["algorithmic_bytes_per_launch"] == b
    assert roof["achieved"] == pytest.approx(b / 100e-6 / 1e9) and roof["frac"] == pytest.approx(roof["achieved"] / 5000.0)
    assert kern["g_op"]["hbm_frac"] == pytest.approx(480 / 7.5e-6 / 1e9 / 5000.0)
    kern, roof = bench.roofline(stats, 1000, 10, 5000.0, "measured", deterministic=True)
    assert roof["kernel"] == "adj_p2g_gather" and roof["achieved"] is None and roof["frac"] is None
    assert roof["traffic"] is None  # the recorded figure is the float kernel's
    assert not any("hbm_frac" in v for v in kern.values())
    assert bench.roofline({}, 1000, 10, 5000.0, "measured", deterministic=False) == ({}, None)
