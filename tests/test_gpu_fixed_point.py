"""FP64 transforms run in 64-bit fixed point scaled per line: accuracy over
lengths, dynamic range and scale, and lines without a finite result.

Tolerance: per pass ~0.6 2^-53 of the r.m.s. at the longest line, three passes,
plus numpy's own FP64 transform (~1e-15): 4e-15 relative L2."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
TOL = 4e-15


def _forward(ctx, x):
    import monofonic_gb300 as mf
    g = mf.Grid_FFT(ctx, x.shape[0], 1.0, "f64")
    g.set_real(x)
    g.FourierTransformForward()
    k = g.get_k()
    g.FourierTransformBackward()
    return k, g.get_real()


@pytest.mark.parametrize("n", [16, 32, 64, 96, 128, 192])
@pytest.mark.parametrize("kind", ["white", "steep", "spike", "lines"])
def test_transform_accuracy(ctx, n, kind):
    rng = np.random.default_rng(n)
    x = rng.standard_normal((n, n, n))
    if kind == "steep":
        k1 = np.fft.fftfreq(n) * n
        k2 = k1[:, None, None] ** 2 + k1[None, :, None] ** 2 + np.arange(n // 2 + 1)[None, None, :] ** 2
        k2[0, 0, 0] = 1.0
        x = np.fft.irfftn(np.fft.rfftn(x) / k2 ** 2, s=(n, n, n), axes=(0, 1, 2))
    elif kind == "spike":
        x = np.zeros((n, n, n))
        x[3, n // 2, n - 1] = -1.7
    elif kind == "lines":  # neighbouring lines 2^-300 .. 2^300 apart
        x = np.ldexp(x, rng.integers(-300, 301, size=(n, n, 1)))
    k, back = _forward(ctx, x)
    want = np.fft.rfftn(x) / np.sqrt(float(n) ** 3)
    assert np.linalg.norm(k - want) <= TOL * np.linalg.norm(want)
    assert np.linalg.norm(back - x) <= 2 * TOL * np.linalg.norm(x)


@pytest.mark.parametrize("n", [16, 96, 128])
@pytest.mark.parametrize("shift", [-990, -700, 700, 990])
def test_scale_does_not_matter(ctx, n, shift):
    x = np.random.default_rng(5).standard_normal((n, n, n))
    k0, b0 = _forward(ctx, x)
    k1, b1 = _forward(ctx, np.ldexp(x, shift))
    # beyond the range that the norm is summed in, the scale comes from the
    # largest value: a few bits fewer
    k1 = np.ldexp(k1.real, -shift) + 1j * np.ldexp(k1.imag, -shift)
    assert np.linalg.norm(k1 - k0) <= 8 * TOL * np.linalg.norm(k0)
    assert np.linalg.norm(np.ldexp(b1, -shift) - x) <= 8 * TOL * np.linalg.norm(x)


@pytest.mark.parametrize("n", [32, 96])
def test_zero_and_non_finite(ctx, n):
    x = np.zeros((n, n, n))
    k, b = _forward(ctx, x)
    assert not k.any() and not b.any()
    x = np.random.default_rng(1).standard_normal((n, n, n))
    for bad in (np.nan, np.inf):
        y = x.copy()
        y[1, 2, 3] = bad
        k, b = _forward(ctx, y)
        assert not np.isfinite(k).any() and not np.isfinite(b).any()
