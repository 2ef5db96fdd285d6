"""The draining wave (a small run in one launch, its daughters appended to the queue it reads) against
the same histories in waves with the post-step kernel: the same tracks on the same random numbers, so
equal counts and tallies to FP64 summation order.  Sizes about a lane, a warp, one track to a warp,
one to a lane, and more; a queue that its daughters outgrow; every scoring instance."""
import numpy as np
import pytest

from moquimc_gb300 import beamline as bl
from moquimc_gb300 import capi
from moquimc_gb300 import phantom as ph
from moquimc_gb300 import workloads

pytestmark = pytest.mark.gpu

COUNTS = ("steps", "histories", "tracks", "secondaries", "local_daughters", "dropped")
NXYZ, LXYZ = (40, 40, 110), (80.0, 80.0, 220.0)


def _box(make, debug, shifter=False):
    c = make()
    c.set_physics(debug)
    if shifter:
        bl.range_shifter((-60.0, -60.0, 10.0), (60.0, 60.0, 25.0), 1.19).add_to(c)
    cid = c.add_child(*ph.phantom_box_edges(LXYZ, (0.0, 0.0, -110.0), NXYZ))
    c.set_hu(cid, np.zeros(NXYZ[::-1], np.int16))
    return c, cid


def _same(a, b):
    for x, y in zip(a[0], b[0]):
        np.testing.assert_allclose(x, y, rtol=1e-9, atol=1e-300)
    assert [a[1][k] for k in COUNTS if k != "tracks"] == [b[1][k] for k in COUNTS if k != "tracks"]


def _run(c, ids, v, mode):
    c.set_post_step_mode(mode)
    c.set_vertices(v)
    c.reset()
    c.transport(0, len(v), 41)
    return [c.tally(i) for i in ids], c.stats()


@pytest.mark.parametrize("debug", [False, True])
@pytest.mark.parametrize("n", [1, 2, 33, 607, 1825, 3041, 58_368, 58_369, 60_001, 97_281])
def test_sizes(gpu_ctx_factory, n, debug):
    c, cid = _box(gpu_ctx_factory, debug)
    ids = [c.add_scorer(cid, capi.DOSE_W)]
    v = ph.uniform_spot_vertices(n, np.random.default_rng(n), 160.0, (0.0, 0.0, 0.5), (30.0, 30.0))
    got, ref = _run(c, ids, v, -1), _run(c, ids, v, 1)
    _same(got, ref)
    assert got[1]["waves"] == 1 and got[1]["tracks"] == n + got[1]["secondaries"]


@pytest.mark.parametrize("chunk, waves", [(0, 1), (700, 2)])
def test_daughters_that_outgrow_the_queue_wait_for_the_next_wave(gpu_ctx_factory, chunk, waves):
    """Two children and debug physics: every deposit-only daughter is queued, dozens to a primary, and
    a queue of 2100 entries does not hold them all."""
    c, cid = _box(gpu_ctx_factory, True, shifter=True)
    ids = [c.add_scorer(cid, capi.EDEP)]
    v = ph.uniform_spot_vertices(60, np.random.default_rng(5), 150.0, (0.0, 0.0, 60.0), (20.0, 20.0))
    ref = _run(c, ids, v, 1)
    assert 2100 < 60 + ref[1]["secondaries"] < 4200
    if chunk:
        c = _box(gpu_ctx_factory, True, shifter=True)[0]
        ids = [c.add_scorer(1, capi.EDEP)]
        c.set_tuning(primary_chunk=chunk)
    got = _run(c, ids, v, -1)
    _same(got, ref)
    assert got[1]["waves"] == waves


@pytest.mark.parametrize("block, per_sm", [(32, 1), (128, 4), (256, 2), (128, 6), (256, 64)])
@pytest.mark.parametrize("n", [1, 1201])
def test_ordinary_waves_in_every_shape(gpu_ctx_factory, n, block, per_sm):
    c, cid = _box(gpu_ctx_factory, False)
    ids = [c.add_scorer(cid, capi.DOSE_W)]
    v = ph.uniform_spot_vertices(n, np.random.default_rng(n), 150.0, (0.0, 0.0, 0.5), (30.0, 30.0))
    ref = _run(c, ids, v, 1)
    c.set_tuning(block=block, blocks_per_sm=per_sm)
    got = _run(c, ids, v, 1)
    _same(got, ref)
    assert got[1]["waves"] == ref[1]["waves"]


def _contour(rng):
    m = rng.random(int(np.prod(NXYZ))) < 0.5
    edge = np.flatnonzero(np.diff(np.concatenate([[0], m.view(np.int8), [0]])))
    stride = (edge[1::2] - edge[0::2]).astype(np.uint32)
    return {"roi_method": capi.ROI_CONTOUR, "start": edge[0::2].astype(np.uint32), "stride": stride,
            "acc": np.cumsum(stride).astype(np.uint32)}


@pytest.mark.parametrize("n", [4001, 80_003])
@pytest.mark.parametrize("scorers", ["edep", "pair", "two", "let", "contour", "let_contour"])
def test_scoring_instances(gpu_ctx_factory, scorers, n):
    c, cid = _box(gpu_ctx_factory, False)
    roi = _contour(np.random.default_rng(8)) if "contour" in scorers else {}
    if scorers == "edep":
        ids = [c.add_scorer(cid, capi.EDEP)]
    else:
        ids = [c.add_scorer(cid, capi.DOSE_W, **roi)]
    if scorers == "pair":
        ids += list(c.add_stat_scorers(cid))
    if scorers == "two":
        ids.append(c.add_scorer(cid, capi.EDEP_PRIMARY))
    if scorers.startswith("let"):
        ids += [c.add_scorer(cid, t, **roi) for t in (capi.LETD_NUM, capi.LETD_DEN)]
    v = ph.uniform_spot_vertices(n, np.random.default_rng(9), 140.0, (0.0, 0.0, 0.5), (30.0, 30.0))
    _same(_run(c, ids, v, -1), _run(c, ids, v, 1))


def test_dij_and_scenarios(gpu_ctx_factory):
    sp = workloads.spot_plan(3, 1, 8.0, 0.5, 4.0, (90.0, 150.0), (300.0, 900.0))
    res = []
    for mode in (-1, 1):
        c, cid = _box(gpu_ctx_factory, False)
        c.set_post_step_mode(mode)
        dij = c.add_dij_scorer(cid, capacity=1 << 20)
        n = c.set_spot_plan(sp)
        c.transport_plan(0, n, 19)
        res.append(c.dij_build(dij).csr())
        d, did = _box(gpu_ctx_factory, False)
        d.set_post_step_mode(mode)
        e = [ph.phantom_box_edges(LXYZ, (0.7 * k, 0.0, -110.0), NXYZ) for k in range(3)]
        d.set_scenarios(did, [x[0] for x in e], [x[1] for x in e], [x[2] for x in e], [1.0, 1.035, 0.965])
        ids = [d.add_scorer(did, capi.DOSE_W)]
        d.set_spot_plan(sp)
        d.transport_plan(0, n, 19)
        res[-1] += (d.tally(ids[0]), d.stats()["steps"])
    for x, y in zip(*res):
        np.testing.assert_allclose(x, y, rtol=2.0 ** -23, atol=1e-300)


@pytest.mark.parametrize("mode", [-1, 1])
@pytest.mark.parametrize("capacity", [1 << 21, 1 << 13])
def test_dij_alone_instance(gpu_ctx_factory, mode, capacity):
    """A Dij scorer by itself runs an instance of its own; beside a dense scorer it takes the generic
    scoring loop.  The same matrix from a sparse table and from one that is mostly full."""
    sp = workloads.spot_plan(2, 2, 6.0, 0.5, 3.0, (60.0, 90.0), (300.0, 700.0))
    csr = []
    for extra in (False, True):
        c, cid = _box(gpu_ctx_factory, False)
        c.set_post_step_mode(mode)
        dij = c.add_dij_scorer(cid, capacity=capacity)
        if extra:
            c.add_scorer(cid, capi.EDEP)
        n = c.set_spot_plan(sp)
        c.transport_plan(0, n, 23)
        csr.append(c.dij_build(dij).csr())
    np.testing.assert_array_equal(csr[0][0], csr[1][0])
    np.testing.assert_array_equal(csr[0][1], csr[1][1])
    np.testing.assert_allclose(csr[0][2], csr[1][2], rtol=2.0 ** -23, atol=0)
    assert csr[0][0][-1] > capacity // 2 or capacity > 1 << 13


@pytest.mark.parametrize("shifter", [False, True])
@pytest.mark.parametrize("debug", [False, True])
def test_a_track_is_counted_once(gpu_ctx_factory, debug, shifter):
    """Resumed after a nuclear interaction or a slice, a track is not another one: primaries and queued
    daughters, whatever the waves."""
    n = 3000
    v = ph.uniform_spot_vertices(n, np.random.default_rng(3), 160.0, (0.0, 0.0, 60.0), (30.0, 30.0))
    for mode, slices, streamed in ((-1, 0, 1), (0, 0, 0), (1, 0, 1), (1, 0, 0), (1, 7, 1), (-1, 7, 0)):
        c, cid = _box(gpu_ctx_factory, debug, shifter)
        c.add_scorer(cid, capi.EDEP)
        c.set_tuning(slice_steps=slices)
        c.set_launch_mode(streamed)
        _, st = _run(c, [], v, mode)
        assert st["tracks"] == n + st["secondaries"], (mode, slices, streamed)
        assert st["secondaries"] > 0
