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


@pytest.mark.parametrize("n", [16, 32, 96, 256])
@pytest.mark.parametrize("size", [1e12, 1e200])
def test_dropped_imaginary_parts_do_not_count(ctx, n, size):
    """A c2r ignores the imaginary parts of its lines' kz = 0 and, unless the
    lines are padded, kz = N/2 values, so however large they are the result
    keeps every bit.  The modes (0, 0, 0) and (0, 0, N/2) have columns of their
    own."""
    import monofonic_gb300 as mf
    L = 50.0
    rng = np.random.default_rng(n)
    s = rng.standard_normal((n, n, n // 2 + 1)) + 1j * rng.standard_normal((n, n, n // 2 + 1))
    s[:, :, 0] = 0
    s[:, :, n // 2] = 0
    g = mf.Grid_FFT(ctx, n, L, "f64", "k")
    h = mf.Grid_FFT(ctx, n, L, "f64", "k")
    out = mf.Grid_FFT(ctx, n, L, "f64", "k")
    padded, aliased = mf.OrszagConvolver(ctx, n, L, "f64"), mf.NaiveConvolver(ctx, n, L, "f64")
    h.set_k(s)
    res = []
    for im in (0.0, size):
        one = []
        s[0, 0, 0] = 1j * im
        g.set_k(s)
        padded.multiply_field(g, h, mf.op.assign_to(out))
        one.append(out.get_k())
        s[0, 0, n // 2] = 1j * im
        g.set_k(s)
        aliased.multiply_field(g, h, mf.op.assign_to(out))
        one.append(out.get_k())
        g.FourierTransformBackward()
        one.append(g.get_real())
        res.append(one)
    for a, b in zip(*res):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("n", [16, 96, 128])
@pytest.mark.parametrize("shift", [-1030, -1060])
def test_subnormal_values_count(ctx, n, shift):
    """A field of subnormal values is transformed like any other.  Every pass
    rounds its results to the subnormal spacing 2^-1074: half of it per
    component, at the last pass (the earlier ones' grow less than the values)
    2^-1075 sqrt(2) of a field of r.m.s. 2^shift; four times that is allowed."""
    import monofonic_gb300 as mf
    x = np.ldexp(np.random.default_rng(n).standard_normal((n, n, n)), shift)
    g = mf.Grid_FFT(ctx, n, 1.0, "f64")
    g.set_real(x)
    g.FourierTransformForward()
    k = g.get_k()
    up = np.ldexp(k.real, -shift) + 1j * np.ldexp(k.imag, -shift)
    want = np.fft.rfftn(np.ldexp(x, -shift)) / np.sqrt(float(n) ** 3)
    tol = 4e-15 + 4 * np.sqrt(2.0) * np.ldexp(1.0, -1075 - shift)
    assert np.linalg.norm(up - want) <= tol * np.linalg.norm(want)
    g.FourierTransformBackward()
    back = np.ldexp(g.get_real(), -shift)
    assert np.linalg.norm(back - np.ldexp(x, -shift)) <= 2 * tol * np.linalg.norm(np.ldexp(x, -shift))


@pytest.mark.parametrize("n", [16, 32, 96, 128, 192])
@pytest.mark.parametrize("kind", ["white", "spike", "lines"])
def test_powers_of_two_factor_out(ctx, n, kind):
    """Values times a power of two give results times that power, bit for bit,
    as FP64 arithmetic does: the scale follows the line's norm however far it
    is from 1, and whatever the lines beside it hold."""
    import monofonic_gb300 as mf
    rng = np.random.default_rng(n)
    x = rng.standard_normal((n, n, n))
    if kind == "spike":
        x = np.zeros((n, n, n))
        x[3, n // 2, n - 1], x[1, 2, 3] = -1.7, 0.3
    elif kind == "lines":  # neighbouring lines 2^-100 .. 2^100 apart
        x = np.ldexp(x, rng.integers(-100, 101, size=(n, n, 1)))
    g = mf.Grid_FFT(ctx, n, 1.0, "f64")
    h, out = mf.Grid_FFT(ctx, n, 1.0, "f64", "k"), mf.Grid_FFT(ctx, n, 1.0, "f64", "k")
    cv = mf.OrszagConvolver(ctx, n, 1.0, "f64")

    def run(shift):
        g.set_real(np.ldexp(x, shift))
        g.FourierTransformForward()
        k = g.get_k()
        h.set_k(np.ldexp(k.real, -shift // 2) + 1j * np.ldexp(k.imag, -shift // 2))
        cv.multiply_field(h, h, mf.op.assign_to(out))
        p = out.get_k()
        g.FourierTransformBackward()
        return [np.ldexp(a, -shift) for a in (k.real, k.imag, g.get_real(), p.real, p.imag)]

    want = run(0)
    for shift in (-400, -130, -104, 120, 400):
        for a, b in zip(run(shift), want):
            assert np.array_equal(a, b), shift


# relative L2 that FP64 butterflies leave of the product below, measured
BUTTERFLIES = {64: 3.1e-16, 96: 3.6e-16, 128: 5.0e-16, 192: 5.5e-16, 256: 3.4e-16, 384: 3.8e-16, 512: 5.8e-16}


@pytest.mark.parametrize("n", list(BUTTERFLIES))
@pytest.mark.parametrize("amp", [8, 12, 13])
def test_products_are_as_accurate_as_butterflies(ctx, n, amp):
    """A product with a field of one mode is the other field shifted both ways:
    exact sums of 53-bit values here but for the normalisation.  The error of the
    fixed-point lines depends on the amplitude (the scale is a power of two)."""
    import monofonic_gb300 as mf
    rng = np.random.default_rng(n)
    h = n // 2
    s = np.zeros((n, n, h + 1), complex)
    s.real[:, :, 1:h] = rng.integers(-2 ** 48, 2 ** 48, size=(n, n, h - 1))
    s.imag[:, :, 1:h] = rng.integers(-2 ** 48, 2 ** 48, size=(n, n, h - 1))
    s[h] = s[:, h] = 0
    s *= amp
    f, g, out = (mf.Grid_FFT(ctx, n, 1.0, "f64", "k") for _ in range(3))
    f.set_k(s)
    q = np.zeros_like(s)
    q[1, 1, 0] = q[-1, -1, 0] = 1
    g.set_k(q)
    mf.OrszagConvolver(ctx, n, 1.0, "f64").multiply_field(f, g, mf.op.assign_to(out))
    got = out.get_k()
    want = (np.roll(s, (1, 1), (0, 1)) + np.roll(s, (-1, -1), (0, 1))) / np.sqrt(float(n) ** 3)
    for a in (got, want):
        a[h] = a[:, h] = a[:, :, h] = 0
    assert np.linalg.norm(got - want) <= BUTTERFLIES[n] * np.linalg.norm(want)


@pytest.mark.parametrize("n, trials", [(16, 40), (32, 40), (64, 20), (96, 10), (128, 6), (192, 3), (256, 2), (512, 1)])
def test_coherent_lines_do_not_overflow(ctx, n, trials):
    """Lines whose values add up in phase reach the bound that the scale is set
    by: single waves forward, single cells backward, and the product of two
    cells' fields, at amplitudes all over an octave.  An overflow is an error
    of order one; the bound is that of the other accuracy tests."""
    import monofonic_gb300 as mf
    rng = np.random.default_rng(n)
    g, out = mf.Grid_FFT(ctx, n, 1.0, "f64"), mf.Grid_FFT(ctx, n, 1.0, "f64", "k")
    cvs = [c(ctx, n, 1.0, "f64") for c in (mf.OrszagConvolver, mf.NaiveConvolver)]
    h = n // 2
    norm = np.linalg.norm

    def wave(p, sign, phase):
        """exp(i sign (p . index) 2 pi / n + i phase)"""
        a = [np.exp(1j * sign * ((p[d] * np.arange(n)) % n) * (2 * np.pi / n)) for d in range(3)]
        return a[0][:, None, None] * a[1][None, :, None] * a[2][None, None, :] * np.exp(1j * phase)

    for trial in range(trials):
        amp, phase = 2 ** rng.uniform(0, 1), rng.integers(0, 8) * np.pi / 4
        if trial % 2 == 0:  # a single mode at the top of a scale (1.3125 / 1.015625), its components equal
            amp, phase = 1.2922, np.pi / 4 + (trial // 2) % 4 * np.pi / 2
        b = rng.integers(0, n, 3)
        b[2] = rng.integers(1, h)
        g.set_real(amp * wave(b, 1, phase).real)
        g.FourierTransformForward()
        k = g.get_k()
        want = np.zeros_like(k)
        want[tuple(b)] = amp / 2 * np.exp(1j * phase) * np.sqrt(float(n) ** 3)
        assert norm(k - want) <= 4e-15 * norm(want)
        g.set_k(want)
        g.FourierTransformBackward()
        want = amp * wave(b, 1, phase).real
        assert norm(g.get_real() - want) <= 4e-15 * norm(want)
        # a cell: every mode has the same modulus (cells on even sites: the Nyquist planes are real)
        p = 2 * rng.integers(0, h, 3)
        cell = amp * wave(p, -1, 0.0)[:, :, : h + 1]
        g.set_k(cell)
        g.FourierTransformBackward()
        r = g.get_real()
        want = np.zeros_like(r)
        want[tuple(p)] = amp * np.sqrt(float(n) ** 3)
        assert norm(r - want) <= 4e-15 * norm(want)
        g.set_k(cell)
        cvs[1].multiply_field(g, g, mf.op.assign_to(out))
        want = cell * (amp * np.sqrt(float(n) ** 3))
        assert norm(out.get_k() - want) <= 8e-15 * norm(want)
        cell[h] = cell[:, h] = cell[:, :, h] = 0  # padded: the modes with |K - k| < N/2 on every axis add up
        g.set_k(cell)
        cvs[0].multiply_field(g, g, mf.op.assign_to(out))
        count = n - 1 - np.abs(np.fft.fftfreq(n) * n)
        want = cell * (amp / np.sqrt(float(n) ** 3)) * (
            count[:, None, None] * count[None, :, None] * count[None, None, : h + 1])
        assert norm(out.get_k() - want) <= 8e-15 * norm(want)
        g.set_real(np.zeros((n, n, n)))
