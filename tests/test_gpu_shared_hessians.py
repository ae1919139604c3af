"""The six padded Hessians from three x transforms (shared sources) against one
convolution per term: phi(2), phi(3) and A(3) of 3LPT and phi(2) of 2LPT.

Tolerance: both forms leave ~5e-16 (FP64) and ~5e-7 (FP32) of a source; the
bounds are those of the other comparisons of the two forms."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
TOL = {"f64": 1e-12, "f32": 1e-5}


@pytest.mark.parametrize("prec", ["f64", "f32"])
@pytest.mark.parametrize("n, order", [(16, 3), (32, 2), (64, 3), (96, 3), (128, 2), (192, 2)])
def test_shared_hessians(ctx, n, order, prec):
    from monofonic_gb300 import ic
    sc = ic.cosmology_scalars(ic.Cosmology(), 24.0)
    out = {}
    for per_term in (False, True):
        cfg = ic.ICConfig(ngrid=n, boxlen=1.7 * n, zstart=24.0, lpt_order=order, precision=prec, out_kind="fields",
                          per_term_conv=per_term)
        gen = ic.ICGenerator(ctx, cfg, sc)
        gen.set_noise_seed(9)
        gen.run(to_host=False)
        out[per_term] = [gen.potential(w) for w in range(1, 6 if order == 3 else 2)]
        gen.close()
    k1 = np.fft.fftfreq(n) * n
    k2 = k1[:, None, None] ** 2 + k1[None, :, None] ** 2 + np.arange(n // 2 + 1)[None, None, :] ** 2
    for a, b in zip(out[False], out[True]):  # k^2 times a potential is its source
        assert np.linalg.norm((a - b) * k2) < TOL[prec] * np.linalg.norm(b * k2)
