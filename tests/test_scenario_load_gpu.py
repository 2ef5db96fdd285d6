"""Robust runs whose scenarios outnumber the entries of a queue load (any chunk is accepted): a load then
holds one history's scenarios, and none of them may be lost.  Against the default chunk."""
import numpy as np
import pytest

from moquimc_gb300 import capi
from moquimc_gb300 import phantom as ph

pytestmark = pytest.mark.gpu

NXYZ, LXYZ = (20, 20, 60), (60.0, 60.0, 120.0)


def _run(make, n_scen, n, chunk, streamed):
    c = make()
    c.set_physics(False)
    e = [ph.phantom_box_edges(LXYZ, (0.05 * k, 0.0, -60.0), NXYZ) for k in range(n_scen)]
    cid = c.add_child(*e[0])
    c.set_scenarios(cid, [x[0] for x in e], [x[1] for x in e], [x[2] for x in e], [1.0 + 0.001 * k for k in range(n_scen)])
    c.set_hu(cid, np.zeros(NXYZ[::-1], np.int16))
    sid = c.add_scorer(cid, capi.EDEP)
    c.set_tuning(primary_chunk=chunk)
    c.set_launch_mode(streamed)
    c.set_vertices(ph.uniform_spot_vertices(n, np.random.default_rng(6), 90.0, (0.0, 0.0, 0.5), (10.0, 10.0)))
    c.transport(0, n, 12)
    return c.tally(sid), c.stats()


@pytest.mark.parametrize("streamed", [0, 1])
@pytest.mark.parametrize("n_scen, n, chunk", [(4, 9, 1), (21, 5, 6), (64, 3, 1), (64, 3, 21), (64, 3, 22)])
def test_no_scenario_is_lost(gpu_ctx_factory, n_scen, n, chunk, streamed):
    want, ref = _run(gpu_ctx_factory, n_scen, n, 1 << 21, 1)
    got, st = _run(gpu_ctx_factory, n_scen, n, chunk, streamed)
    assert st["histories"] == ref["histories"] == n * n_scen and st["steps"] == ref["steps"]
    assert (want.reshape(n_scen, -1).sum(axis=1) > 0).all()
    np.testing.assert_allclose(got, want, rtol=1e-9, atol=1e-300)
