"""Robust scenarios whose edge arrays are shared, all different, or too long for a block's shared memory,
against one context per scenario: the same tracks, so tallies equal to FP64 summation order."""
import numpy as np
import pytest

from moquimc_gb300 import capi
from moquimc_gb300 import phantom as ph

pytestmark = pytest.mark.gpu

LXYZ = (60.0, 60.0, 120.0)


@pytest.mark.parametrize("nxyz, shifts", [
    ((20, 21, 60), [(0, 0, 0), (3, 0, 0), (0, 3, 0), (0, 0, 0), (3, 3, -3)]),
    ((20, 21, 60), [(0.1 * k, -0.2 * k, 0.3 * k) for k in range(7)]),
    ((400, 300, 1500), [(0, 0, 0), (0, 0, 2)]),
    ((600, 400, 2000), [(0, 0, 0), (1, 0, 0), (0, 1, 2)]),
])
def test_scenarios_equal_their_own_runs(gpu_ctx_factory, nxyz, shifts):
    n = 150
    v = ph.uniform_spot_vertices(n, np.random.default_rng(2), 60.0, (0.0, 0.0, 3.5), (10.0, 10.0))
    hu = np.zeros(nxyz[::-1], np.int16)
    edges = [ph.phantom_box_edges(LXYZ, (s[0], s[1], s[2] - 60.0), nxyz) for s in shifts]
    scale = [1.0 + 0.02 * (k % 2) for k in range(len(shifts))]
    with capi.Context(0) as c:
        c.set_physics(False)
        cid = c.add_child(*edges[0])
        c.set_scenarios(cid, [e[0] for e in edges], [e[1] for e in edges], [e[2] for e in edges], scale)
        c.set_hu(cid, hu)
        sid = c.add_scorer(cid, capi.EDEP)
        c.set_vertices(v)
        c.transport(0, n, 8)
        got = c.tally(sid).reshape(len(shifts), -1)
    for k, e in enumerate(edges):
        with capi.Context(0) as d:
            d.set_physics(False)
            did = d.add_child(*e)
            d.set_hu(did, hu, scale[k])
            s = d.add_scorer(did, capi.EDEP)
            d.set_vertices(v)
            d.transport(0, n, 8)
            want = d.tally(s)
        assert want.sum() > 0
        np.testing.assert_allclose(got[k], want, rtol=1e-9, atol=1e-300)
