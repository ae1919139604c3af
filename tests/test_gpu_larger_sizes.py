"""Aliased products at N=384 against a 64-bit product, and the six Hessians
from three x transforms at N=256 and 384 against one convolution per term.

Tolerances: those of the same comparisons at the smaller sizes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
TOL = {"f64": 1e-12, "f32": 1e-5}


@pytest.mark.parametrize("prec", ["f64", "f32"])
@pytest.mark.parametrize("nop", [2, 3])
def test_aliased_products_384(ctx, prec, nop):
    import monofonic_gb300 as mf
    from oracle import lpt_oracle as O
    n, L = 384, 100.0
    spec = [O.r2c(np.random.default_rng(20 + i).standard_normal((n, n, n))) for i in range(nop)]
    g = [mf.Grid_FFT(ctx, n, L, prec, "k") for _ in range(nop)]
    out = mf.Grid_FFT(ctx, n, L, prec, "k")
    for a, s in zip(g, spec):
        a.set_k(s)
    dirs = [(0, 0), (1, 2), (2, 2)][:nop]
    args = [x for pair in zip(g, dirs) for x in pair]
    mf.NaiveConvolver(ctx, n, L, prec).convolve_Hessians(*args, mf.op.assign_to(out))
    want = (O.naive_conv2, O.naive_conv3)[nop - 2](*(O.hessian(s, L, *d) for s, d in zip(spec, dirs)))
    assert np.linalg.norm(out.get_k() - want) < TOL[prec] * np.linalg.norm(want)


@pytest.mark.parametrize("n, prec", [(256, "f64"), (256, "f32"), (384, "f32")])
def test_shared_hessians(ctx, n, prec):
    from tests.test_gpu_shared_hessians import test_shared_hessians as compare
    compare(ctx, n, 3, prec)
