"""Compute_PowerSpectrum's bins against numpy: counts exactly, sums to FP64
rounding (tolerance: n^3 terms of one sign added in any order, 1e-12)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [16, 32, 96, 128, 192])
@pytest.mark.parametrize("prec", ["f64", "f32"])
@pytest.mark.parametrize("box", [100.0, 317.3])
def test_bins(ctx, n, prec, box):
    import monofonic_gb300 as mf
    g = mf.Grid_FFT(ctx, n, box, prec)
    g.fill_white_noise(17)
    k, P, eP, cnt = g.Compute_PowerSpectrum()
    z = g.get_k().astype(np.complex128)
    kf = 2.0 * np.pi / box
    idx = np.arange(n)
    k1 = (idx - n * (idx > n // 2)).astype(np.float64) * kf
    kz = np.arange(n // 2 + 1).astype(np.float64) * kf
    kk = np.sqrt((k1[:, None, None] ** 2 + k1[None, :, None] ** 2) + kz[None, None, :] ** 2)
    ok = (kk >= kf) & (kk < kf * (n // 2))
    b = (kk[ok] / kf).astype(int)
    w = np.broadcast_to(np.where(np.arange(n // 2 + 1) == 0, 1.0, 2.0), kk.shape)[ok]
    nb = len(k)
    want = np.bincount(b, weights=w, minlength=nb)[:nb]
    assert np.array_equal(cnt, want.astype(np.int64))
    has = want > 0
    v = (z.real ** 2 + z.imag ** 2)[ok]
    f = box ** 3 / (2 * np.pi) ** 3 / float(n) ** 3
    wp = np.bincount(b, weights=w * v, minlength=nb)[:nb][has] / want[has] * f
    wk = np.bincount(b, weights=w * kk[ok], minlength=nb)[:nb][has] / want[has]
    assert np.allclose(P[has], wp, rtol=1e-12, atol=0) and np.allclose(k[has], wk, rtol=1e-12, atol=0)
