"""The per-voxel material tables follow what they are made from: after each call that changes a density
or a curve, a context that has transported before gives the tallies of one that has not."""
import numpy as np
import pytest

from moquimc_gb300 import capi
from moquimc_gb300 import phantom as ph

pytestmark = pytest.mark.gpu

N, LXYZ, NXYZ = 1500, (60.0, 60.0, 150.0), (30, 31, 75)
EDGES = ph.phantom_box_edges(LXYZ, (0.0, 0.0, -75.0), NXYZ)


def _calib():
    return capi.CalibTable.sample(lambda rho, e: 1.05, lambda rho: 0.3 / max(rho, 1e-4), 0.0, 1e-4, 32, 0.5, 10.0, 24)


def _scenarios(c, scales):
    e = [ph.phantom_box_edges(LXYZ, (0.4 * k, 0.0, -75.0), NXYZ) for k in range(len(scales))]
    c.set_scenarios(0, [x[0] for x in e], [x[1] for x in e], [x[2] for x in e], scales)


def _hu(seed):
    return np.random.default_rng(seed).integers(-900, 1200, NXYZ[::-1]).astype(np.int16)


# each step changes one thing of the context's state
STEPS = [
    lambda c: c.set_hu(0, _hu(1)),
    lambda c: c.set_hu(0, _hu(2), 1.035),
    lambda c: c.set_density(0, np.random.default_rng(3).uniform(2e-4, 2e-3, NXYZ[::-1]).astype(np.float32)),
    lambda c: c.set_physics(True),
    lambda c: c.set_calibration(_calib()),
    lambda c: c.set_calibration(None),
    lambda c: _scenarios(c, [1.0, 0.965]),
    lambda c: _scenarios(c, [1.035, 1.0, 1.035]),
    lambda c: _scenarios(c, []),
]


def _context(make):
    c = make()
    c.set_physics(False)
    c.add_child(*EDGES)
    c.set_vertices(ph.uniform_spot_vertices(N, np.random.default_rng(7), 120.0, (0.0, 0.0, 0.5), (15.0, 15.0)))
    return c, c.add_scorer(0, capi.DOSE_W)


@pytest.mark.parametrize("last", range(len(STEPS)))
def test_tables_follow_their_sources(gpu_ctx_factory, last):
    c, sid = _context(gpu_ctx_factory)
    f, fid = _context(gpu_ctx_factory)
    for k in range(last + 1):
        STEPS[k](c)
        STEPS[k](f)
        if k < last:
            c.transport(0, N, 5)      # builds the tables that the next step has to drop
    c.reset()
    c.transport(0, N, 11)
    f.transport(0, N, 11)
    np.testing.assert_allclose(c.tally(sid), f.tally(fid), rtol=1e-9, atol=1e-300)
    assert c.stats()["steps"] == f.stats()["steps"] > 0
