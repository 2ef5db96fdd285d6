"""What a context sets up -- tables, tallies, curves, edges, plans -- is ordered with its own stream, whatever
the legacy stream still has to do: work queued there (a caller's, on torch's default stream) must not
come between a setup call and the first work that reads its result."""
import numpy as np
import pytest

from moquimc_gb300 import capi

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
