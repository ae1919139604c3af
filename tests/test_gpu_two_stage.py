"""FP32 strided passes in two stages (pass lengths 128..768) against the
FP64 transforms: every output operator of a padded product, the N-grid
transforms, and a 3LPT run, whose pair products go through the truncation pass.

Tolerance: a transform of these lengths leaves ~1.2e-7 per pass in FP32, nine
passes in quadrature ~4e-7 of the result; 3e-6 is several times that."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
TOL = 3e-6


def _rel(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


def _potential(ctx, n, prec):
    import monofonic_gb300 as mf
    g = mf.Grid_FFT(ctx, n, float(n), prec)
    g.fill_white_noise(11)
    g.apply_InverseLaplacian()
    return g


# passes of length N (N-grid) and 3N/2 (padded): 96/144, 128/192, 192/288, 256/384, 384/576, 512/768
@pytest.mark.parametrize("n", [96, 128, 192, 256, 384, 512])
def test_products_and_transforms(ctx, n):
    import monofonic_gb300 as mf
    out = {}
    for prec in ("f32", "f64"):
        phi = _potential(ctx, n, prec)
        o = mf.Grid_FFT(ctx, n, float(n), prec, "k")
        cv = mf.OrszagConvolver(ctx, n, float(n), prec)
        cv.convolve_SumOfHessians(phi, (0, 0), phi, (1, 1), (2, 2), mf.op.assign_to(o))
        cv.convolve_Hessians(phi, (0, 1), phi, (0, 2), mf.op.add_to(o))
        cv.convolve_Hessians(phi, (1, 2), phi, (1, 2), mf.op.subtract_from(o))
        cv.convolve_Gradients(phi, (0,), phi, (2,), mf.op.multiply_add_to(o, -0.3))
        k = o.get_k()
        o.FourierTransformBackward()
        out[prec] = (k, o.get_real())
        del cv, o, phi
    assert _rel(out["f32"][0], out["f64"][0]) < TOL
    assert _rel(out["f32"][1], out["f64"][1]) < TOL


@pytest.mark.parametrize("n", [96, 128, 192])
def test_truncated_pairs(ctx, n):
    from monofonic_gb300 import ic
    sc = ic.cosmology_scalars(ic.Cosmology(), 24.0)
    phi3 = {}
    for prec in ("f32", "f64"):
        cfg = ic.ICConfig(ngrid=n, boxlen=2.0 * n, zstart=24.0, lpt_order=3, precision=prec, out_kind="fields")
        gen = ic.ICGenerator(ctx, cfg, sc)
        gen.set_noise_seed(5)
        gen.run(to_host=False)
        phi3[prec] = [gen.potential(w) for w in (2, 3)]
        gen.close()
    k1 = np.fft.fftfreq(n) * n
    k2 = k1[:, None, None] ** 2 + k1[None, :, None] ** 2 + np.arange(n // 2 + 1)[None, None, :] ** 2
    for a, b in zip(phi3["f32"], phi3["f64"]):
        # the sources (k^2 times the potential): the potential's lowest modes cancel
        assert _rel(a * k2, b * k2) < TOL
