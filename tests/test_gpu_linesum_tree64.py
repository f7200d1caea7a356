"""The interpolated FP64 line sum (uniform grids) against the kernel that evaluates every
line at every point, which takes the same call when its grid is not uniform: two extra
points at irregular steps send the whole grid there, and the common points are compared.

Tolerance.  Every term of the sum is non-negative (H falls below its value at the cutoff
nowhere inside it), so errors add relative to the sum itself.  One line's interpolation
error is below 6e-16 of its largest value on its block, which is at most
((1.85 + 1) / (1.85 - 1))^2 = 11.3 of its smallest there; carrying 32 node values down two
levels and to the points adds a few rounding errors times the weights' absolute sum (about
3 per level).  1e-12 of the point's value leaves a factor of ten over that and over the
rounding of 5,000-term sums on both sides.  Where a point is reached only by lines within
a hair of their cutoff, H and its pedestal cancel to rounding: 1e-15 of the peak covers it.
"""
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


def _both(pkg, ctx, ll, grid, T, p, **kw):
    tree = pkg.compute_voigt_cross_sections(grid, ll, T, p, backend=ctx, **kw)
    step = grid[-1] - grid[-2] if len(grid) > 1 else 0.01
    odd = np.concatenate([grid, grid[-1] + step * np.array([0.37, 5.11])])
    direct = pkg.compute_voigt_cross_sections(odd, ll, T, p, backend=ctx, **kw)[:-2]
    assert np.all(np.abs(tree - direct) <= 1e-12 * np.abs(direct) + 1e-15 * direct.max()), \
        np.max(np.abs(tree - direct) / (np.abs(direct) + 1e-3 * direct.max()))
    assert direct.max() > 0.0


# edges of lanes, rows, leaves, groups and strips of 32-point leaves; the last takes
# 128-point leaves (from 302,977 points of one layer)
@pytest.mark.parametrize("n", [1, 2, 31, 33, 128, 129, 511, 513, 2047, 5501, 302977])
def test_sizes(pkg, ctx, n):
    ll = pkg.synthetic.synthetic_linelist(1500, 2, 31, 640.0, 720.0)
    grid = 660.0 + np.arange(n) * (0.0025 if n < 10000 else 0.0002)
    _both(pkg, ctx, ll, grid, 250.0, 0.3)


@pytest.mark.parametrize("p", [0.0, 1e-6, 0.02, 1.0])
@pytest.mark.parametrize("method,cutoff,x_far", [
    ("FullFaddeeva", 25.0, 122.0), ("FullFaddeeva", 0.03, 122.0), ("FullFaddeeva", 1.3, 122.0),
    ("FullFaddeeva", 25.0, 5.0), ("FullFaddeeva", 25.0, 1e5), ("Weideman", 25.0, 122.0)])
def test_methods_and_windows(pkg, ctx, p, method, cutoff, x_far):
    """Pressures from none to the surface's, cutoffs narrower than a leaf, a strip and the
    usual one, cores from nearly none to wider than the cutoff."""
    ll = pkg.synthetic.synthetic_linelist(700, 2, 32, 640.0, 720.0)
    grid = 650.0 + np.arange(9001) * 0.005
    _both(pkg, ctx, ll, grid, 220.0, p, method=pkg.VoigtMethod[method], cutoff=cutoff, x_far=x_far)


@pytest.mark.parametrize("nu_lo,step,n", [(2500.0, 0.0025, 20001), (1300.0, 0.02, 3001), (700.0, 1.0, 300)])
def test_other_ranges(pkg, ctx, nu_lo, step, n):
    """Wide Doppler cores, a coarse grid (a leaf wider than the core) and a step of 1 cm^-1
    (leaves wider than the cutoff)."""
    ll = pkg.synthetic.synthetic_linelist(800, 1, 33, nu_lo - 20.0, nu_lo + n * step + 20.0)
    _both(pkg, ctx, ll, nu_lo + np.arange(n) * step, 290.0, 0.9, vmr_self=0.02)


def test_few_lines_and_rounded_grid(pkg, ctx):
    ll = pkg.synthetic.synthetic_linelist(1, 2, 34, 660.0, 661.0)
    _both(pkg, ctx, ll, 655.0 + np.arange(4001) * 0.0025, 250.0, 0.3)
    # grid points a few ulp off the uniform grid, as linspace and range arithmetic leave them
    g = np.random.Generator(np.random.PCG64(1))
    ll = pkg.synthetic.synthetic_linelist(900, 2, 35, 640.0, 720.0)
    grid = 660.0 + np.arange(5000) * 0.0025
    _both(pkg, ctx, ll, grid + 3e-13 * g.standard_normal(len(grid)), 250.0, 0.3)


def test_line_mixing_small_grid(pkg, ctx, oracle, orc_mod):
    """VP_Y on a grid short enough for 32-point leaves against the FP64 oracle (the wider
    forward cases of test_gpu_parity.py take 128-point leaves): BT within 1e-6 K, as there."""
    ll = pkg.synthetic.synthetic_linelist(1200, 2, 36, 670.0, 720.0)
    y0 = pkg.synthetic.vpy_y0(len(ll), seed=37)
    prof = pkg.afgl_atmosphere("us_standard")
    snd = pkg.Sounder.make(695.0, 697.0, 0.25, opd_max=2.0, fwhm_gauss=0.5)
    kw = dict(internal_dnu=0.0025, apply_continuum=False, with_ils=False)
    _, _, bt = pkg.forward_model(prof, {2: ll}, sounder=snd, backend=ctx, precision="fp64",
                                 line_mixing=pkg.VPYLineMixing(y0), **kw)
    ref = oracle.forward_model(dict(p=prof.pressure, T=prof.temperature, vmr=prof.vmr), {2: ll.lines},
                               orc_mod.sounder(695.0, 697.0, 0.25, opd_max=2.0, fwhm_gauss=0.5),
                               orc_mod.fm_options(line_mixing=True, **kw), y0={2: y0})[1]
    assert np.max(np.abs(bt - ref)) < 1e-6
