"""The Jacobian's channel contraction takes two state elements at a time: an odd and an even
number of them, one and several channel tiles, every column against the stand-alone convolution
(irs_apply_ils) of the monochromatic Jacobian.

Tolerance: FP32 taps, products and sums: one rounding per tap and product and at most
12801 / 100 + 15 < 160 terms in a row per thread, 32 + 8 partial sums: (160 + 40 + 3) 2^-24 =
1.3e-5 of sum |D| |tap|."""
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


@pytest.mark.parametrize("emissivity", [False, True])
@pytest.mark.parametrize("n_ch", [1, 15, 16, 50])
def test_every_column(pkg, ctx, emissivity, n_ch):
    lists = {2: pkg.synthetic.synthetic_linelist(300, 2, 41, 690.0, 740.0)}
    prof = pkg.afgl_atmosphere("tropical")
    prof = pkg.AtmosphericProfile(prof.pressure[::10], prof.temperature[::10], prof.altitude[::10],
                                  {s: v[::10] for s, v in prof.vmr.items()})
    lo, hi = 700.0, 700.0 + (n_ch - 1) * 0.25
    snd = pkg.Sounder.make(lo, hi, 0.25, opd_max=2.0, fwhm_gauss=0.5)
    mono = pkg.Sounder.make(lo - 16.0, hi + 16.0, 0.0025, opd_max=2.0, fwhm_gauss=0.5)
    spec = pkg.StateVectorSpec(len(prof.pressure), [pkg.CO2], include_emissivity=emissivity)
    kw = dict(backend=ctx, apply_continuum=False, observable="radiance", eps_sfc=0.95)
    K = pkg.analytic_jacobian(prof, lists, spec, sounder=snd, high_res_factor=100, **kw).K
    D = pkg.analytic_jacobian(prof, lists, spec, sounder=mono, high_res_factor=1, with_ils=False, **kw).K
    _, taps = pkg.ils_kernel(0.0025, 2.0, 0.5, backend=ctx)
    at = len(taps) // 2 + 100 * np.arange(n_ch)
    nu = lo - 16.0 + 0.0025 * np.arange(D.shape[0])
    assert K.shape == (n_ch, spec.n)
    for x in range(spec.n):
        ref = pkg.apply_ils(nu, D[:, x], None, taps, backend=ctx)[at]
        most = pkg.apply_ils(nu, np.abs(D[:, x]), None, np.abs(taps), backend=ctx)[at]
        assert np.all(np.abs(K[:, x] - ref) <= 1.3e-5 * most + 1e-30), x
