"""The tuner's candidates: a scoring mode whose wave comes in one launch shape is not timed once per shape,
and the setting it had stays."""
import numpy as np
import pytest

from moquimc_gb300 import capi
from moquimc_gb300 import workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scorers, shapes", [("edep", 4), ("two", 4), ("pair", 1), ("let", 1)])
def test_candidates(gpu_ctx_factory, scorers, shapes):
    wl = workloads.c2(histories=3000)
    c = gpu_ctx_factory()
    c.set_physics(False)
    cid = c.add_child(*wl.edges())
    c.set_hu(cid, wl.hu)
    c.add_scorer(cid, {"let": capi.LETT_NUM, "edep": capi.EDEP}.get(scorers, capi.DOSE_W))
    if scorers == "two":
        c.add_scorer(cid, capi.EDEP)
    if scorers == "pair":
        c.add_stat_scorers(cid)
    c.set_tuning(block=96, blocks_per_sm=7)
    c.set_vertices(wl.vertices(3000, 8))
    res = c.autotune(0, 3000, 9)
    assert len(res) == 2 * shapes          # two launch modes, one queue size: all exceed the sample
    assert len(np.unique(res[["block", "blocks_per_sm", "streamed"]])) == len(res)
    if shapes == 1:
        assert set(res["block"]) == {96} and set(res["blocks_per_sm"]) == {7}
