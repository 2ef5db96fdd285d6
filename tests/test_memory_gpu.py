"""A context's optional memory -- the material tables -- never costs a call the memory it cannot do without:
tables are refused where they would take most of what is free, and given back when another allocation
needs their place, in the middle of a run too.  The rest of the device's memory is held by an allocation
of the test's; tallies do not depend on whether there is a table."""
import numpy as np
import pytest

from moquimc_gb300 import capi
from moquimc_gb300 import phantom as ph
from moquimc_gb300 import workloads

pytestmark = pytest.mark.gpu

MB = 1 << 20
NXYZ, LXYZ = (280, 280, 300), (280.0, 280.0, 300.0)     # a table takes 359 MB, the queues below 51 MB
TABLE = 16 * int(np.prod(NXYZ))
N = 100_000                                             # records of more than 12 MB
MANY = 500_000                                          # of 42 MB and more


def _context(make, nxyz=NXYZ, n=N):
    c = make()
    c.set_physics(False)
    c.set_tuning(primary_chunk=1 << 19 if n == MANY else 1 << 17)
    c.add_child(*ph.phantom_box_edges(LXYZ, (0.0, 0.0, -150.0), nxyz))
    c.set_hu(0, np.zeros(nxyz[::-1], np.int16))
    c.set_vertices(ph.uniform_spot_vertices(n, np.random.default_rng(2), 100.0, (0.0, 0.0, 0.5), (30.0, 30.0)))
    return c, c.add_scorer(0, capi.DOSE_W)


@pytest.fixture
def make():
    """Contexts that are closed with the test."""
    made = []

    def new():
        made.append(capi.Context(0))
        return made[-1]

    yield new
    for c in made:
        c.close()


@pytest.fixture
def fill():
    """fill(leave): hold all but about `leave` bytes of the device's free memory."""
    import torch

    held = []
    # the kernels' code and stacks are on the device before it is full
    with capi.Context(0) as c:
        _context(lambda: c, (28, 28, 30), 200)
        for mode in (-1, 1):
            c.set_post_step_mode(mode)
            c.transport(0, 200, 1)

    def hold(leave):
        torch.cuda.empty_cache()
        free = torch.cuda.mem_get_info()[0]
        held.append(torch.empty(free - leave, dtype=torch.uint8, device="cuda"))
        assert abs(torch.cuda.mem_get_info()[0] - leave) < 4 * MB

    yield hold
    held.clear()
    torch.cuda.empty_cache()


@pytest.fixture(scope="module")
def reference(built_lib):
    with capi.Context(0) as c:
        _, sid = _context(lambda: c)
        c.transport(0, N, 9)
        return c.tally(sid)


def _check(c, sid, reference):
    np.testing.assert_allclose(c.tally(sid), reference, rtol=1e-9, atol=1e-300)


def test_a_table_leaves_room_for_the_records(make, fill, reference):
    c, sid = _context(make)
    fill(TABLE + 56 * MB)
    c.transport(0, N, 9)
    _check(c, sid, reference)


def test_a_table_is_given_back_for_a_tally(make, fill, reference):
    c, sid = _context(make)
    c.transport(0, N, 9)
    fill(16 * MB)
    more = c.add_scorer(0, capi.EDEP)      # 188 MB
    c.reset()
    c.transport(0, N, 9)
    _check(c, sid, reference)
    assert c.tally(more).sum() > 0


@pytest.mark.parametrize("mode", [-1, 1])
def test_a_table_is_given_back_within_a_run(make, fill, mode):
    c, sid = _context(make, n=MANY)
    c.transport(0, MANY, 9)
    want = c.tally(sid)
    c.close()
    c, sid = _context(make, n=MANY)
    c.set_post_step_mode(mode)
    c.transport(0, 1000, 9)                # the table, the queues, the smallest record array: 5.5 MB
    c.reset()
    fill(24 * MB)
    c.transport(0, MANY, 9)
    _check(c, sid, want)


def test_a_refused_table_is_tried_again(make, reference):
    import torch

    c, sid = _context(make)
    torch.cuda.empty_cache()
    c.transport(0, 1, 9)                   # the queues and the records are there, and a table
    c.set_physics(True)
    c.set_physics(False)                   # drops it
    free = torch.cuda.mem_get_info()[0]
    held = torch.empty(free - TABLE - 64 * MB, dtype=torch.uint8, device="cuda")
    c.transport(0, 1, 9)
    del held
    torch.cuda.empty_cache()
    c.reset()
    before = torch.cuda.mem_get_info()[0]
    c.transport(0, N, 9)
    _check(c, sid, reference)
    assert before - torch.cuda.mem_get_info()[0] > 0.9 * TABLE


def test_a_reset_frees_a_large_matrix(make):
    import torch

    c = make()
    c.set_physics(False)
    nxyz = (200, 200, 200)
    c.add_child(*ph.phantom_box_edges((200.0, 200.0, 200.0), (0.0, 0.0, -100.0), nxyz))
    c.set_hu(0, np.zeros(nxyz[::-1], np.int16))
    sid = c.add_dij_scorer(0, capacity=1 << 27)
    total = c.set_spot_plan(workloads.spot_plan(20, 18, 8.0, 0.5, 4.0, (120.0, 150.0), (18_000.0, 22_000.0)))
    c.transport_plan(0, total, 3)
    assert c.dij_build(sid).nnz * 16 > 1.1 * 512 * MB      # at least 14 bytes an entry, and 6 a voxel row
    before = torch.cuda.mem_get_info()[0]
    c.reset()
    assert torch.cuda.mem_get_info()[0] - before > 512 * MB
    c.transport_plan(0, int(c.plan_cum[3]), 3)
    assert c.dij_build(sid).csr()[0][-1] > 0
