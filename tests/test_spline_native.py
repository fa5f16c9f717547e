"""The native not-a-knot spline against scipy's, from the fewest points on.

Tolerance: the tridiagonal system is diagonally dominant inside (its inverse
amplifies an error below 1) and well conditioned at the ends for knots whose
spacings differ by less than 4: a few dozen roundings of the largest
coefficient times its power of the spacing.
"""
import numpy as np
import pytest


@pytest.mark.parametrize("n", [4, 5, 6, 7, 33, 1000])
@pytest.mark.parametrize("even", [True, False])
def test_spline_matches_scipy(n, even):
    from scipy.interpolate import CubicSpline
    from dftpy_gb300._tables import spline_notaknot
    rng = np.random.default_rng(n)
    x = np.cumsum(np.full(n, 0.5) if even else rng.uniform(0.25, 1.0, n))
    y = rng.standard_normal(n)
    xs, c = spline_notaknot(x, y)
    ref = CubicSpline(x, y, bc_type="not-a-knot").c[::-1].T        # (a, b, c, d) rows
    assert c.shape == (n - 1, 4) and np.array_equal(xs, x)
    np.testing.assert_allclose(c, ref, rtol=0, atol=256 * 2.0 ** -53 * np.abs(ref).max())


def test_spline_refuses():
    from dftpy_gb300._tables import spline_notaknot
    with pytest.raises(ValueError):
        spline_notaknot(np.arange(3.0), np.arange(3.0))
    with pytest.raises(ValueError):
        spline_notaknot(np.arange(5.0), np.arange(4.0))
