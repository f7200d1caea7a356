"""Positions within the Faddeeva core of the FP32 line sum (IRS_MIXED), in every row of a leaf,
against the FP64 sum of the same call.

Tolerances.  d is a difference of exact and nearly exact terms, so x = d fx and y carry the rounding
of fx and y (6e-8 each) and their products (6e-8 each): x^2 within 4e-7, and the quotient of
|x| + y >= 15 with its five roundings and the reciprocal's ulp within 1.5e-6 of its value with the
two-level fraction's own 2e-7; 5e-7 of the peak is the FP32 Faddeeva's bound nearer the centre.
Doppler cores: a relative error e of x changes exp(-x^2) by 2 x^2 exp(-x^2) e < 0.8 e of the peak,
1e-6 of the peak with the Faddeeva's 5e-7 and some overlapping lines."""
import numpy as np
import pytest

from conftest import load_package

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def pkg():
    return load_package()


@pytest.fixture(scope="module")
def ctx(pkg):
    c = pkg.B200Context()
    yield c
    c.close()


def both(pkg, ctx, ll, grid, T, p, **kw):
    return [pkg.compute_voigt_cross_sections(grid, ll, T, p, backend=ctx, precision=q, **kw) for q in ("mixed", "fp64")]


@pytest.mark.parametrize("row", range(8))
@pytest.mark.parametrize("p", [1e-6, 3e-5, 3e-4, 2e-3])
@pytest.mark.parametrize("x_far", [122.0, 0.2])
def test_narrow_lines(pkg, ctx, row, p, x_far):
    """Lines in the far infrared, x = 110 per step: centres a fraction of a step past a point."""
    step = 0.0005
    grid = 4.0 + np.arange(2000) * step
    ll = pkg.synthetic.synthetic_linelist(1, 2, 91, 4.0, 5.0).lines.copy()
    ll["pressure_shift"] = 0.0
    for off in (0.14, 0.3, 0.45):
        ll["wavenumber"] = 4.0 + step * (1024 + 32 * row + 13 + off)
        got, ref = both(pkg, ctx, pkg.HITRANLinelist(ll), grid, 300.0, p, x_far=x_far)
        assert np.all(np.abs(got - ref) <= 1.5e-6 * ref + 5e-7 * ref.max()), np.max(np.abs(got / ref - 1))


@pytest.mark.parametrize("p", [0.0, 1e-9, 1e-6])
def test_crowded_doppler_cores(pkg, ctx, p):
    """More inner points per tile than the buffer holds (sixty lines per leaf)."""
    ll = pkg.synthetic.synthetic_linelist(2400, 1, 92, 544.0, 557.0).lines.copy()
    ll["intensity"] = 1e-21
    ll["lower_energy"] = 100.0
    got, ref = both(pkg, ctx, pkg.HITRANLinelist(ll), 545.0 + np.arange(4000) * 0.0025, 200.0, p)
    assert np.max(np.abs(got - ref)) <= 1e-6 * ref.max()
