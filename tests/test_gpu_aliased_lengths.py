"""Aliased products (include/convolution.hh:296-420) at grid sizes whose fused z
pass takes other line batches than the powers of two, against the oracle.

Tolerance: the FP32 forward and inverse passes leave ~5e-7 of the product, the
FP64 ones ~1e-15; the bounds are those of the other convolution tests."""
import numpy as np
import pytest

from oracle import lpt_oracle as O

pytestmark = pytest.mark.gpu
TOL = {"f64": 1e-12, "f32": 1e-5}


def _rel(a, b):
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


@pytest.mark.parametrize("prec", ["f64", "f32"])
@pytest.mark.parametrize("n", [96, 128, 192])
def test_aliased_products(ctx, n, prec):
    import monofonic_gb300 as mf
    L = 100.0
    spec = [O.r2c(np.random.default_rng(20 + i).standard_normal((n, n, n))) for i in range(3)]
    g = [mf.Grid_FFT(ctx, n, L, prec, "k") for _ in range(3)]
    out = mf.Grid_FFT(ctx, n, L, prec, "k")
    for a, s in zip(g, spec):
        a.set_k(s)
    cv = mf.NaiveConvolver(ctx, n, L, prec)
    cv.convolve_Hessians(g[0], (0, 0), g[1], (1, 2), mf.op.assign_to(out))
    ref = O.naive_conv2(O.hessian(spec[0], L, 0, 0), O.hessian(spec[1], L, 1, 2))
    assert _rel(out.get_k(), ref) < TOL[prec]
    cv.convolve_Hessians(g[0], (0, 0), g[1], (1, 1), g[2], (2, 2), mf.op.assign_to(out))
    ref = O.naive_conv3(*(O.hessian(s, L, d, d) for d, s in enumerate(spec)))
    assert _rel(out.get_k(), ref) < TOL[prec]
