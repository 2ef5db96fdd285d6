"""A run may take any number of queue loads, however small the chunk: the limit on waves, which ends a run
that makes no progress, counts from the last load."""
import numpy as np
import pytest

from moquimc_gb300 import capi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("streamed", [0, 1])
def test_more_loads_than_the_wave_limit(gpu_ctx_factory, streamed):
    n = 200_200
    c = gpu_ctx_factory()
    c.set_physics(False)
    e = np.array([-10.0, 10.0], np.float32)
    c.add_child(e, e, np.array([-10.0, 0.0, 10.0], np.float32))
    c.set_density(0, np.full((2, 1, 1), 1e-3, np.float32))
    sid = c.add_scorer(0, capi.EDEP)
    c.set_tuning(primary_chunk=1)
    c.set_launch_mode(streamed)
    v = np.zeros(n, capi.VERTEX_DTYPE)
    v["ke"], v["pos"], v["dir"] = 0.25, (0.0, 0.0, 5.0), (0.0, 0.0, -1.0)      # below the tracking cut: one step each
    c.set_vertices(v)
    c.transport(0, n, 3)
    st = c.stats()
    assert st["histories"] == n and st["waves"] > 200_000
    np.testing.assert_array_equal(c.tally(sid), [0.0, 0.25 * n])
