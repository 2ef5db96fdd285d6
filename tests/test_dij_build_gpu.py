"""The Dij build (compaction, radix passes, both layouts) on matrices of the sizes where its tiles, its
digits and its kept memory change: against the recorded insertions, and the voxel rows through D.w
with unit weights.  Values: FP64 sums of at most a few hundred insertions in another order, then one
rounding to FP32."""
import numpy as np
import pytest

from moquimc_gb300 import capi
from moquimc_gb300 import phantom as ph
from moquimc_gb300 import workloads

pytestmark = pytest.mark.gpu


def _context(make, nxyz):
    c = make()
    c.set_physics(False)
    cid = c.add_child(*ph.phantom_box_edges((64.0, 64.0, 130.0), (0.0, 0.0, -65.0), nxyz))
    c.set_hu(cid, np.zeros(nxyz[::-1], np.int16))
    return c, cid


def _check(c, dij, n_spots, nxyz):
    vox, spot, val = c.dij_hits(dij)
    op = c.dij_build(dij, n_spots=n_spots)
    indptr, indices, data = op.csr()
    nv = int(np.prod(nxyz))
    key, inv = np.unique(spot.astype(np.int64) * nv + vox, return_inverse=True)
    want = np.bincount(inv, weights=val, minlength=len(key)) if len(key) else np.zeros(0)
    assert op.nnz == len(key) == indptr[-1]
    np.testing.assert_array_equal(indices.astype(np.int64) + np.repeat(np.arange(n_spots), np.diff(indptr)) * nv, key)
    np.testing.assert_allclose(data, want, rtol=2.0 ** -23, atol=0)
    dose = np.zeros(nv)
    np.add.at(dose, key % nv, data.astype(np.float64))
    np.testing.assert_allclose(c.dij_matvec(dij, np.ones(n_spots), nv), dose, rtol=1e-13 * max(1, n_spots // 100), atol=0)
    # FP32: a sum of m positive terms in order is off by at most m roundings
    longest = np.bincount(key % nv).max() if len(key) else 1
    np.testing.assert_allclose(c.dij_matvec(dij, np.ones(n_spots, np.float32), nv), dose, rtol=longest * 2.0 ** -24, atol=0)
    g = np.random.default_rng(1).standard_normal(nv)
    want = np.zeros(n_spots)
    np.add.at(want, key // nv, data.astype(np.float64) * g[key % nv])
    size = np.zeros(n_spots)
    np.add.at(size, key // nv, np.abs(data.astype(np.float64) * g[key % nv]))
    assert (np.abs(c.dij_rmatvec(dij, g, n_spots) - want) <= 1e-12 * size).all()
    return op


@pytest.mark.parametrize("nxyz, spots, per_spot", [((1, 1, 2), 1, 3), ((3, 2, 5), 2, 40), ((16, 16, 65), 5, 200),
                                                   ((64, 64, 130), 9, 300), ((64, 64, 130), 260, 12),
                                                   ((1, 1, 2), 7000, 2), ((2, 2, 5), 66_000, 1)])
def test_build_against_the_recorded_insertions(gpu_ctx_factory, nxyz, spots, per_spot):
    """The last two: rows longer than a stage of the forward, and columns past 16 bits."""
    c, cid = _context(gpu_ctx_factory, nxyz)
    dij = c.add_dij_scorer(cid, capacity=1 << 20)
    c.dij_record_hits(dij, 1 << 23)
    sp = workloads.spot_plan(spots, 1, 40.0 / spots, 0.5, 3.0, (60.0, 110.0), (per_spot, per_spot + 1))
    n = c.set_spot_plan(sp)
    c.transport_plan(0, n, 3)
    _check(c, dij, spots, nxyz)


def test_builds_that_follow_one_another(gpu_ctx_factory):
    """Small, large, small, empty and rejected builds of one scorer in the memory the last one left."""
    nxyz = (64, 64, 130)
    c, cid = _context(gpu_ctx_factory, nxyz)
    dij = c.add_dij_scorer(cid, capacity=1 << 20)
    for k, (spots, h) in enumerate([(2, 5), (40, 200), (3, 4), (1, 0), (7, 60)]):
        c.reset()
        c.dij_record_hits(dij, 1 << 22)
        if h:
            n = c.set_spot_plan(workloads.spot_plan(spots, 1, 3.0, 0.5, 3.0, (60.0, 110.0), (h, h + 1)))
            c.transport_plan(0, n, 100 + k)
        _check(c, dij, spots, nxyz)
    with pytest.raises(capi.MqiError) as e:
        c.dij_build(dij, n_spots=6)               # spot 6 has entries
    assert e.value.code == capi.MQI_ERR_INVALID
    with pytest.raises(capi.MqiError) as e:
        c.dij_matvec(dij, np.ones(7), int(np.prod(nxyz)))
    assert e.value.code == capi.MQI_ERR_STATE
    c.dij_build(dij, n_spots=7)
