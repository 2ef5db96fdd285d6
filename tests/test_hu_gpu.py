"""HU -> density on the device at every HU value and the sizes and alignments where the vectorised
conversion changes path, against the C restatement, bit for bit."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def densities(oracle):
    return np.array([oracle.hu_to_density(h) for h in range(-1000, 2996)], np.float32)


@pytest.mark.parametrize("n", [1, 7, 8, 9, 4095, 65536, 1 << 21 | 5])
@pytest.mark.parametrize("skip_hu, skip_rho", [(0, 0), (1, 0), (8, 3), (8, 4)])
def test_hu_to_density_on_device(gpu_ctx_factory, densities, n, skip_hu, skip_rho):
    import torch

    scale = np.float32(1.035)
    hu = np.random.default_rng(n).integers(-32768, 32767, n).astype(np.int16) if n < 4096 else np.resize(
        np.arange(-1100, 3100, dtype=np.int16), n)
    d_hu = torch.zeros(n + skip_hu, dtype=torch.int16, device="cuda")
    d_hu[skip_hu:] = torch.from_numpy(hu)
    d_rho = torch.full((n + skip_rho + 1,), -7.0, dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    c = gpu_ctx_factory()
    c._check(c.lib.mqi_hu_to_density(c.h, C.c_void_p(d_hu.data_ptr() + 2 * skip_hu),
                                     C.c_void_p(d_rho.data_ptr() + 4 * skip_rho), n, C.c_float(scale), 1), c.h)
    got = d_rho.cpu().numpy()
    np.testing.assert_array_equal(got[skip_rho:-1], densities[np.clip(hu, -1000, 2995).astype(int) + 1000] * scale)
    assert (got[:skip_rho] == -7.0).all() and got[-1] == -7.0
