"""FP64 lines in fixed point: the scale of a line is a function of its values
alone."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _in_bin(rng, mag):
    """a value whose bound in the L1 sum is mag, a multiple of 2^-20 of its power
    of two: its upper 20 mantissa bits plus one unit"""
    m, e = np.frexp(mag)  # mag = m 2^e, m in [1/2, 1); the value may lie one binade below
    unit = np.ldexp(1.0, e - 21) if m > 0.5 else np.ldexp(1.0, e - 22)
    return mag - unit * rng.uniform(0.1, 0.9)


@pytest.mark.parametrize("n, tpl, trials", [(96, 3, 24), (192, 6, 6), (384, 12, 2)])
def test_equal_lines_give_equal_results(ctx, n, tpl, trials):
    """A field with modes (0, 0, kz) only has one and the same padded z line
    everywhere, so its square has no mode off that axis: exactly none where
    every line is transformed alike.  The line is one whose bound, summed over
    its tpl threads in FP32, falls on either side of a power of two depending
    on the order of the sum: threads 0 and 1 hold half an ulp each, which is
    lost when added to the last thread's part one by one."""
    import monofonic_gb300 as mf
    L = 100.0
    M = 3 * n // 2
    scale = 1.5 ** 1.5 / np.sqrt(float(M) ** 3)  # the operands' normalisation
    f, out = mf.Grid_FFT(ctx, n, L, "f64", "k"), mf.Grid_FFT(ctx, n, L, "f64", "k")
    cv = mf.OrszagConvolver(ctx, n, L, "f64")
    ulp = np.ldexp(1.0, -23)
    # the largest sum that 65/64 (the rounding margin) keeps below 2
    a, h = np.float32(2064888 * 8 * ulp), np.float32(ulp / 2)
    g = np.float32(65 / 64)
    assert ((h + h) + a) * g >= 2 > ((a + h) + h) * g
    rng = np.random.default_rng(n)
    for _ in range(trials):
        s = np.zeros((n, n, n // 2 + 1), complex)
        s[0, 0, tpl - 1] = _in_bin(rng, 2064888 * 8 * ulp) / scale
        s[0, 0, 0] = _in_bin(rng, ulp / 2) / scale
        s[0, 0, 1] = _in_bin(rng, ulp / 2) / scale
        f.set_k(s)
        cv.multiply_field(f, f, mf.op.assign_to(out))
        r = out.get_k()
        assert r[0, 0].any()
        r[0, 0] = 0
        assert not r.any()


@pytest.mark.parametrize("n", [96, 192])
def test_batch_equals_standalone(ctx, n):
    """a 3LPT run in a batch, replayed, and alone: the same bits"""
    from monofonic_gb300.serve import Batch, Request
    from tests.test_gpu_batch import _same, _standalone
    reqs = [Request(ngrid=n, boxlen=2.0 * n, zstart=24.0, lpt_order=3, precision="f64", seed=7),
            Request(ngrid=32, boxlen=64.0, zstart=24.0, lpt_order=2, precision="f64", seed=8)]
    b = Batch(reqs, nstreams=2)
    for _ in range(2):
        b.run()
        for i, r in enumerate(reqs):
            assert _same(b.particles(i), _standalone(ctx, r)), i
    b.close()
