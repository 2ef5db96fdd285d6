"""The persistent FP32 forward over many runs per block: a stage of its ring, whose values a run multiplies
in place, is refilled by a bulk copy as soon as the run is summed.  Each dose value is a sum of FP32
products in spot order, so numpy gives it bit for bit; repeated, as a refill that overtook a store would
show only now and then."""
import numpy as np
import pytest

from moquimc_gb300 import capi
from moquimc_gb300 import phantom as ph
from moquimc_gb300 import workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_spots", [0, 65_536, 65_537])
def test_forward_bits_over_many_runs(gpu_ctx_factory, n_spots):
    import torch

    nxyz = (128, 128, 200)
    c = gpu_ctx_factory()
    c.set_physics(False)
    cid = c.add_child(*ph.phantom_box_edges((128.0, 128.0, 200.0), (0.0, 0.0, -100.0), nxyz))
    c.set_hu(cid, np.zeros(nxyz[::-1], np.int16))
    sid = c.add_dij_scorer(cid, capacity=1 << 24)
    total = c.set_spot_plan(workloads.spot_plan(8, 6, 8.0, 0.5, 4.0, (100.0, 150.0), (12_000.0, 18_000.0)))
    c.transport_plan(0, total, 3)
    op = c.dij_build(sid, n_spots)
    assert op.nnz > 3_800_000      # about a thousand runs of 4096 entries: several for each resident block
    indptr, voxel, value = op.csr()
    w = np.random.default_rng(1).uniform(0.5, 2.0, op.n_spots).astype(np.float32)
    want = np.zeros(op.n_voxels, np.float32)
    for s in range(op.n_spots):
        a, b = indptr[s], indptr[s + 1]
        if b > a:
            want[voxel[a:b]] += value[a:b] * w[s]
    wt = torch.from_numpy(w).cuda()
    for _ in range(20):
        np.testing.assert_array_equal(op.matvec(wt).cpu().numpy(), want)
