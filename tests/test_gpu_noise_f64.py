"""White noise on FP64 grids: bit for bit the host generator's draws."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,seed", [(16, 0), (64, 12345), (96, 2 ** 64 - 1), (192, 77), (256, 3)])
def test_device_noise_is_the_host_noise(ctx, n, seed):
    import monofonic_gb300 as mf
    from monofonic_gb300 import ic
    g = mf.Grid_FFT(ctx, n, 1.0, "f64")
    g.fill_white_noise(seed)
    assert np.array_equal(g.get_real().view(np.uint64), ic.white_noise(n, seed).view(np.uint64))
