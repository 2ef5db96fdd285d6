"""The statistics sweeps (one launch over all scenarios, the threshold decided on integer images of
the tallies) against numpy on the same tallies: odd grids, one to many scenarios, thresholds from
none to the maximum itself, and both estimators.  Tolerance: sums of at most 1e5 FP64 terms in another
order, 1e5 * 2^-53 ~ 1e-11, against 1e-10."""
import numpy as np
import pytest

from moquimc_gb300 import capi
from moquimc_gb300 import phantom as ph

pytestmark = pytest.mark.gpu


def _run(make, nxyz, n_scen, n=3000):
    c = make()
    c.set_physics(False)
    lxyz = (60.0, 60.0, 120.0)
    edges = ph.phantom_box_edges(lxyz, (0.0, 0.0, -60.0), nxyz)
    cid = c.add_child(*edges)
    if n_scen > 1:
        e = [ph.phantom_box_edges(lxyz, (0.5 * k, 0.0, -60.0), nxyz) for k in range(n_scen)]
        c.set_scenarios(cid, [x[0] for x in e], [x[1] for x in e], [x[2] for x in e], [1.0 + 0.01 * k for k in range(n_scen)])
    c.set_hu(cid, np.zeros(nxyz[::-1], np.int16))
    dose = c.add_scorer(cid, capi.DOSE_W)
    pair = c.add_stat_scorers(cid)
    c.set_vertices(ph.uniform_spot_vertices(n, np.random.default_rng(4), 100.0, (0.0, 0.0, 0.5), (20.0, 20.0)))
    c.transport(0, n, 3)
    return c, dose, pair, n


@pytest.mark.parametrize("nxyz, n_scen", [((1, 1, 3), 1), ((3, 5, 7), 2), ((33, 17, 65), 1), ((31, 9, 25), 21), ((40, 41, 60), 3)])
@pytest.mark.parametrize("threshold", [0.0, 0.5, 0.999, 1.0])
def test_reference_estimator(gpu_ctx_factory, nxyz, n_scen, threshold):
    c, _, (d1, d2), n = _run(gpu_ctx_factory, nxyz, n_scen)
    s1, s2 = (c.tally(d).reshape(n_scen, -1) for d in (d1, d2))
    est = []
    for a, b in zip(s1, s2):
        m = a / n
        mean = m.astype(np.float32)
        sigma = np.sqrt(np.maximum(((b / n - m * m) / (n - 1.0)).astype(np.float32), np.float32(0)))
        sel = (a > 0) & (mean.astype(np.float64) > float(mean.max()) * float(np.float32(threshold)))
        est.append(((sigma[sel] / mean[sel]).astype(np.float64).sum() / sel.sum() if sel.any() else 0.0, int(sel.sum())))
    want = max(est, key=lambda x: x[0])
    got = c.stat_uncertainty(d1, d2, n, threshold)
    assert got[1] == want[1]
    np.testing.assert_allclose(got[0], want[0], rtol=1e-10, atol=0)


@pytest.mark.parametrize("threshold", [0.0, 0.5, 1.0])
def test_batch_estimator(gpu_ctx_factory, threshold):
    c, dose, _, n = _run(gpu_ctx_factory, (33, 17, 65), 1)
    x = []
    for k in range(3):
        c.reset()
        c.transport(0, n, 10 + k)
        x.append(c.tally(dose))
        c.batch_accumulate(dose)
    s1, s2 = sum(x), sum(v * v for v in x)
    mean = s1 / 3.0
    var = np.maximum((s2 / 3.0 - mean * mean) / 2.0, 0.0)
    sel = (s1 > 0) & (mean > mean.max() * float(np.float32(threshold)))
    want = (np.sqrt(var[sel] / 3.0) / mean[sel]).sum() / sel.sum() if sel.any() else 0.0
    got = c.batch_uncertainty(dose, threshold)
    assert got[1:] == (int(sel.sum()), 3)
    np.testing.assert_allclose(got[0], want, rtol=1e-10, atol=0)
