"""The batch's tuner times what its kernels depend on, the sort interval, and leaves
the caller's other launch settings alone."""
import pytest

from tests.test_gpu_batch import _batch, _check, batch_case  # noqa: F401 (fixture)

pytestmark = pytest.mark.gpu


def test_tuner_keeps_the_callers_settings(batch_case):  # noqa: F811
    scs, singles = batch_case
    with _batch(scs) as b:
        b.set_launch(sort_every=5, ctas_per_sm=1, particle_block=128, use_graph=False)
        b.setup()
        assert b.autotune(reps=1) > 0
        cfg = b.launch()
        assert cfg["sort_every"] in (4, 8, 16)
        assert (cfg["ctas_per_sm"], cfg["particle_block"], bool(cfg["use_graph"])) == (1, 128, False)
        _check(b, scs, singles, b.gradient())
