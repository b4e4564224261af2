"""GPU: the transforms of every kind of length (each radix, two to four
stages, a length without a generic plan) through egx_fft2d against numpy, with
columns of very different sizes side by side.

Tolerance: numpy's complex128 transforms err by a few 2^-53 of a column's norm
and the device's by at most as much (their roundings are 2^-59 of a bound that
grows by the radices, three to four stages): 1e-15 of each column, a factor of
three above both.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
TOL = 1e-15


@pytest.mark.parametrize("n0,n1,howmany", [(4, 6, 3), (14, 18, 5), (16, 128, 4), (50, 64, 2), (7, 15, 3), (98, 90, 7),
                                           (240, 250, 3), (256, 360, 5), (378, 24, 9), (486, 16, 3), (10, 512, 17),
                                           (1024, 8, 3), (1050, 12, 2)])
@pytest.mark.parametrize("sign", [-1, 1])
def test_fft2d_every_length(egx_ctx, n0, n1, howmany, sign):
    rng = np.random.default_rng(n0 + n1)
    a = rng.standard_normal((n0, n1, howmany)) + 1j * rng.standard_normal((n0, n1, howmany))
    a *= 10.0 ** np.linspace(-100, 100, howmany)  # each column has its own exponent
    a[..., howmany // 2] = 0
    a[n0 // 3, n1 // 2, howmany // 2] = 1 + 2j    # a single peak
    want = np.fft.fft2(a, axes=(0, 1)) if sign < 0 else np.fft.ifft2(a, axes=(0, 1)) * (n0 * n1)
    got = egx_ctx.fft2d(a.copy(), sign)
    err = np.linalg.norm(got - want, axis=(0, 1)) / np.linalg.norm(want, axis=(0, 1))
    assert err.max() < TOL, err


def test_fft2d_nonfinite_and_zero_columns(egx_ctx):
    """A zero column transforms to exact zeros, a NaN or an infinity spoils
    its own column only."""
    rng = np.random.default_rng(3)
    a = rng.standard_normal((30, 28, 4)) + 1j * rng.standard_normal((30, 28, 4))
    want = egx_ctx.fft2d(a.copy(), -1)
    b = a.copy()
    b[..., 0] = 0
    b[3, 4, 1] = np.nan
    b[5, 6, 2] = 1j * np.inf
    got = egx_ctx.fft2d(b, -1)
    assert not got[..., 0].any()
    assert not np.isfinite(got[..., 1]).any() and not np.isfinite(got[..., 2]).any()
    assert np.array_equal(got[..., 3], want[..., 3])


def test_fft2d_of_subnormal_numbers(egx_ctx):
    """Columns at and below 2^-1022 against the transform of the same columns
    scaled into the normal range. A result is rounded to units of 2^-1074 after
    each of the two passes: half a unit per entry, at most 30 of them summed by
    the second pass, in both parts: (30 + 1) / 2 sqrt(2) < 24 units."""
    rng = np.random.default_rng(5)
    a = rng.standard_normal((30, 28, 4)) + 1j * rng.standard_normal((30, 28, 4))
    down = np.array([1040, 1024, 1018, 1060])
    unit = np.ldexp(1.0, -1074)
    x = np.ldexp(a.real, -down) + 1j * np.ldexp(a.imag, -down)
    back = np.ldexp(x.real, down - 8) + 1j * np.ldexp(x.imag, down - 8)  # exact
    want = np.fft.fft2(back, axes=(0, 1))
    got = egx_ctx.fft2d(x.copy(), -1)
    for c in range(4):
        g = np.ldexp(got[..., c].real, down[c] - 8) + 1j * np.ldexp(got[..., c].imag, down[c] - 8)
        assert np.abs(g - want[..., c]).max() < 24 * np.ldexp(unit, down[c] - 8) + TOL * np.linalg.norm(want[..., c])
