"""Lines of the FP32 line sum (IRS_MIXED) on either side of the rules that class them as core or
general: cores as wide as an eighth of the cutoff and at the largest |x| of the packed quotient
(1.8e5), y as large, and steps of a fraction of the cutoff, against the FP64 sum of the same call.

Tolerance: as the other cross sections of this path, 2e-5 of the peak; and where a coarse grid has
no point near a strong line's centre, the FP32 Faddeeva's own bound, 4.5e-7 of the value at the
centre.  Pressures stay where |z|^6 of the continued fraction is in FP32's range (|z| < 2.6e6)."""
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


def _check(pkg, ctx, ll, grid, T, p, **kw):
    ref = pkg.compute_voigt_cross_sections(grid, ll, T, p, backend=ctx, precision="fp64", **kw)
    got = pkg.compute_voigt_cross_sections(grid, ll, T, p, backend=ctx, precision="mixed", **kw)
    assert ref.max() > 0.0
    centres = np.unique(ll.lines["wavenumber"] + p * ll.lines["pressure_shift"].astype(float))
    centre = pkg.compute_voigt_cross_sections(centres, ll, T, p, backend=ctx, precision="fp64", **kw).max()
    assert np.max(np.abs(got - ref)) <= 2e-5 * ref.max() + 4.5e-7 * centre


@pytest.mark.parametrize("p", [0.0, 1e-6, 0.02, 1.0])
@pytest.mark.parametrize("x_far", [1400.0, 1450.0, 2900.0, 3600.0, 4200.0])  # an eighth of 25 cm^-1: x = 3,900 to 4,300
def test_core_of_an_eighth_of_the_cutoff(pkg, ctx, p, x_far):
    ll = pkg.synthetic.synthetic_linelist(700, 2, 47, 640.0, 720.0)
    _check(pkg, ctx, ll, 650.0 + np.arange(6000) * 0.0025, 220.0, p, x_far=x_far)


@pytest.mark.parametrize("p", [1e-3, 0.1, 1.0, 5.0])  # y = 4 to 2e6
@pytest.mark.parametrize("x_far", [122.0, 1e5, 1.7e5, 2e5])
def test_largest_quotients(pkg, ctx, p, x_far):
    """Narrow lines (far infrared): x = 2e5 is reached well inside the cutoff."""
    ll = pkg.synthetic.synthetic_linelist(60, 2, 48, 0.5, 4.0)
    _check(pkg, ctx, ll, 1.0 + np.arange(5000) * 0.0005, 300.0, p, x_far=x_far)


@pytest.mark.parametrize("step,n", [(0.02, 300), (0.05, 2000), (0.1, 110), (0.1, 2000), (0.19, 500), (0.2, 500), (0.5, 300)])
@pytest.mark.parametrize("p", [1e-6, 0.1, 1.0])
def test_coarse_steps(pkg, ctx, step, n, p):
    ll = pkg.synthetic.synthetic_linelist(900, 2, 49, 640.0, 660.0 + n * step)
    _check(pkg, ctx, ll, 650.0 + np.arange(n) * step, 250.0, p)


@pytest.mark.parametrize("x_far", [122.0, 2900.0])
@pytest.mark.parametrize("dnu", [0.0025, 0.05])
def test_line_mixing(pkg, ctx, x_far, dnu):
    """VP_Y (the dispersive part of the quotient), BT of FP32 sums against FP64: 1e-3 K, the path's
    bound."""
    ll = pkg.synthetic.synthetic_linelist(1200, 2, 50, 670.0, 720.0)
    y0 = pkg.synthetic.vpy_y0(len(ll), seed=51)
    snd = pkg.Sounder.make(690.0, 700.0, 0.25, opd_max=2.0, fwhm_gauss=0.5)
    bt = [pkg.forward_model(pkg.afgl_atmosphere("us_standard"), {2: ll}, sounder=snd, backend=ctx, precision=q, internal_dnu=dnu,
                            x_far=x_far, apply_continuum=False, line_mixing=pkg.VPYLineMixing(y0))[2] for q in ("fp64", "mixed")]
    assert np.max(np.abs(bt[1] - bt[0])) < 1e-3
