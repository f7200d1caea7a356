"""The FP32 line sum on the block tree (IRS_MIXED) at the edges of its blocks (leaves of 128
points, strips of 4096), with narrow cutoffs, extreme cores and pressures, against the FP64
sum of the same call.

Tolerances, as for the other cross sections of this path: the FP32 Faddeeva is within 4.5e-7
of a line's centre value, its parameters and positions add a few 1e-7 of it, interpolation
1.6e-8 of a wing, and some tens of lines overlap: 2e-5 of the peak (Weideman-24 in FP32: 5e-5)."""
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


def _check(pkg, ctx, ll, grid, T, p, tol=2e-5, **kw):
    ref = pkg.compute_voigt_cross_sections(grid, ll, T, p, backend=ctx, precision="fp64", **kw)
    got = pkg.compute_voigt_cross_sections(grid, ll, T, p, backend=ctx, precision="mixed", **kw)
    assert ref.max() > 0.0
    assert np.max(np.abs(got - ref)) <= tol * ref.max(), np.max(np.abs(got - ref)) / ref.max()


@pytest.mark.parametrize("n", [2, 127, 128, 129, 257, 4095, 4096, 4097, 12000])
def test_sizes(pkg, ctx, n):
    ll = pkg.synthetic.synthetic_linelist(1500, 2, 41, 640.0, 720.0)
    _check(pkg, ctx, ll, 660.0 + np.arange(n) * 0.0025, 250.0, 0.3)


@pytest.mark.parametrize("p", [1e-6, 0.02, 1.0])
@pytest.mark.parametrize("method,cutoff,x_far", [
    ("FullFaddeeva", 25.0, 122.0), ("FullFaddeeva", 0.2, 122.0), ("FullFaddeeva", 2.0, 122.0),
    ("FullFaddeeva", 25.0, 6.0), ("FullFaddeeva", 25.0, 3000.0), ("Weideman", 25.0, 122.0)])
def test_methods_and_windows(pkg, ctx, p, method, cutoff, x_far):
    ll = pkg.synthetic.synthetic_linelist(700, 2, 42, 640.0, 720.0)
    _check(pkg, ctx, ll, 650.0 + np.arange(9001) * 0.005, 220.0, p, tol=2e-5 if method == "FullFaddeeva" else 5e-5,
           method=pkg.VoigtMethod[method], cutoff=cutoff, x_far=x_far)


@pytest.mark.parametrize("nu_lo,step,n,mol", [(2600.0, 0.0025, 9000, 1), (1300.0, 0.02, 3001, 2), (100.0, 0.001, 9000, 1),
                                              (700.0, 0.0002, 20000, 2)])
def test_other_ranges(pkg, ctx, nu_lo, step, n, mol):
    """Doppler cores from a fifth of a point to several leaves wide."""
    ll = pkg.synthetic.synthetic_linelist(800, mol, 43, nu_lo - 20.0, nu_lo + n * step + 20.0)
    _check(pkg, ctx, ll, nu_lo + np.arange(n) * step, 290.0, 0.9, vmr_self=0.02)


def test_one_line(pkg, ctx):
    ll = pkg.synthetic.synthetic_linelist(1, 2, 44, 660.0, 661.0)
    _check(pkg, ctx, ll, 640.0 + np.arange(20001) * 0.0025, 250.0, 0.3)


def test_empty_windows_give_zero(pkg, ctx):
    """A grid that no line reaches, on either side of the list."""
    ll = pkg.synthetic.synthetic_linelist(50, 2, 45, 800.0, 801.0)
    for lo in (700.0, 900.0):
        s = pkg.compute_voigt_cross_sections(lo + np.arange(5000) * 0.0025, ll, 250.0, 0.3, backend=ctx, precision="mixed")
        assert np.all(s == 0.0)


def test_warp_and_block_trees_agree(pkg, ctx):
    """A grid long enough for one warp per (strip, segment) (2,368 strips of a profile's
    segments: 49 strips x 49 layers) against the windows of it that take eight: BT within the
    1e-4 K that FP32 sums in another order and the window's own lines leave."""
    lists = {2: pkg.synthetic.synthetic_linelist(9000, 2, 46, 645.0, 1190.0)}
    prof = pkg.afgl_atmosphere("us_standard")
    kw = dict(backend=ctx, internal_dnu=0.0025, precision="mixed", apply_continuum=False)
    wide = pkg.Sounder.make(680.0, 1160.0, 0.25, opd_max=2.0, fwhm_gauss=0.5)
    _, _, bt = pkg.forward_model(prof, lists, sounder=wide, **kw)
    for lo in (700.0, 1100.0):
        snd = pkg.Sounder.make(lo, lo + 20.0, 0.25, opd_max=2.0, fwhm_gauss=0.5)
        _, _, b = pkg.forward_model(prof, lists, sounder=snd, **kw)
        k = round((lo - 680.0) / 0.25)
        assert np.max(np.abs(bt[k:k + len(b)] - b)) < 1e-4
