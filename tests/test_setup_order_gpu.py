"""What a context sets up -- tables, tallies, curves, edges, plans -- is ordered with its own stream, whatever
the legacy stream still has to do: work queued there (a caller's, on torch's default stream) must not
come between a setup call and the first work that reads its result."""
import numpy as np
import pytest

from moquimc_gb300 import capi
from moquimc_gb300 import phantom as ph
from moquimc_gb300 import workloads

pytestmark = pytest.mark.gpu


@pytest.fixture
def busy():
    """Queues some tens of milliseconds of copies on the legacy stream."""
    import torch

    a = torch.zeros(1 << 28, dtype=torch.float32, device="cuda")
    b = torch.empty_like(a)
    b.copy_(a)
    torch.cuda.synchronize()

    def queue():
        for _ in range(100):
            b.copy_(a)

    yield queue
    torch.cuda.synchronize()


def test_hu_table_of_a_new_context(busy, oracle):
    want = np.array([oracle.hu_to_density(h) for h in range(-1000, 2996)], np.float32)
    hu = np.arange(-1000, 2996, dtype=np.int16)
    for _ in range(3):
        busy()
        with capi.Context(0) as c:
            np.testing.assert_array_equal(c.hu_to_density(hu), want)
            assert c.stats()["device_errors"] == 0 and c.stats()["steps"] == 0


NXYZ, LXYZ, N = (40, 40, 110), (80.0, 80.0, 220.0), 400
EDGES = ph.phantom_box_edges(LXYZ, (0.0, 0.0, -110.0), NXYZ)


def _calib():
    return capi.CalibTable.sample(lambda rho, e: 1.05, lambda rho: 0.3 / max(rho, 1e-4), 0.0, 1e-4, 32, 0.5, 10.0, 24)


def _roi():
    return {"roi_method": capi.ROI_CONTOUR, "start": [0, 60_000], "stride": [50_000, 90_000], "acc": [50_000, 140_000]}


def _scenarios(c):
    e = [ph.phantom_box_edges(LXYZ, (0.4 * k, 0.0, -110.0), NXYZ) for k in range(2)]
    c.set_scenarios(0, [x[0] for x in e], [x[1] for x in e], [x[2] for x in e], [1.0, 1.035])


# what comes right before a transport, which reads it from the context's stream
SETUPS = {
    "scorer": lambda c: [c.add_scorer(0, capi.DOSE_W)],
    "contour": lambda c: [c.add_scorer(0, capi.DOSE_W, **_roi())],
    "pair": lambda c: list(c.add_stat_scorers(0)),
    "calibration": lambda c: c.set_calibration(_calib()),
    "scenarios": _scenarios,
    "plan": lambda c: c.set_spot_plan(workloads.spot_plan(2, 1, 8.0, 0.5, 4.0, (70.0, 120.0), (200.0, 300.0))),
    "tuning": lambda c: c.autotune(0, N, 3),
}


def _context(make):
    c = make()
    c.set_physics(False)
    c.add_child(*EDGES)
    c.set_hu(0, np.zeros(NXYZ[::-1], np.int16))
    c.set_vertices(ph.uniform_spot_vertices(N, np.random.default_rng(7), 120.0, (0.0, 0.0, 0.5), (15.0, 15.0)))
    ids = [c.add_scorer(0, capi.EDEP)]
    c.transport(0, N, 5)          # the queues and records are there
    c.reset()
    return c, ids


def _transport(c, setup):
    if setup == "plan":
        c.transport_plan(0, c.plan_histories, 11)
    else:
        c.transport(0, N, 11)


@pytest.mark.parametrize("setup", list(SETUPS))
def test_setup_right_before_a_transport(gpu_ctx_factory, busy, setup):
    import torch

    want, ids = _context(gpu_ctx_factory)
    new = SETUPS[setup](want)
    ids += new if isinstance(new, list) else []
    torch.cuda.synchronize()
    _transport(want, setup)
    c, _ = _context(gpu_ctx_factory)
    busy()
    SETUPS[setup](c)
    _transport(c, setup)
    torch.cuda.synchronize()
    for i in ids:
        assert want.tally(i).sum() > 0
        np.testing.assert_allclose(c.tally(i), want.tally(i), rtol=1e-9, atol=1e-300)
    a, b = c.stats(), want.stats()
    assert all(a[k] == b[k] for k in ("histories", "steps", "secondaries")) and a["steps"] > 0
