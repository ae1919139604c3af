"""White noise on FP32 grids: the float-pair evaluation gives exactly the
FP64 generator's draws rounded to the nearest float."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,seed", [(16, 0), (32, 2 ** 63 + 5), (96, 7), (256, 1), (256, 0xFFFFFFFFFFFFFFFF), (384, 20240607)])
def test_fp32_noise_is_the_rounded_fp64_noise(ctx, n, seed):
    import monofonic_gb300 as mf
    g64 = mf.Grid_FFT(ctx, n, 1.0, "f64")
    g32 = mf.Grid_FFT(ctx, n, 1.0, "f32")
    g64.fill_white_noise(seed)
    g32.fill_white_noise(seed)
    want, got = g64.get_real().astype(np.float32), g32.get_real()
    # bit patterns, so that the sign of a zero counts too
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32))
