"""The ILS at channels that are grid nodes (ils_nodes_kernel, jg_channel_nodes_kernel)
against the stand-alone convolution (irs_apply_ils) of the monochromatic spectrum, which
the same call gives when its sounder is the padded internal grid itself.

Tolerances: the spectrum's sums are FP64 over at most 12,801 taps in both, in another
order: 1e-12 relative.  K's are FP32 with FP32 taps: one rounding per tap and product and
at most M = taps/step + 15 <= 816 terms in a row per thread, so (816 + 3) 2^-24 = 4.9e-5
of sum |D| |tap| bounds it."""
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


# (channel step, internal step in cm^-1): the smallest and largest node step of the kernel's
# range (16, 256), a phase count that is and is not a multiple of 32, and 15 (the general kernel)
@pytest.mark.parametrize("dnu,factor", [(0.25, 15), (0.25, 16), (0.25, 32), (0.5, 50), (0.25, 100), (0.625, 125),
                                        (1.0, 256)])
@pytest.mark.parametrize("n_ch", [1, 8, 17])
def test_spectrum_and_jacobian(pkg, ctx, dnu, factor, n_ch):
    lists = {2: pkg.synthetic.synthetic_linelist(300, 2, 41, 690.0, 740.0)}
    prof = pkg.afgl_atmosphere("tropical")
    prof = pkg.AtmosphericProfile(prof.pressure[::7], prof.temperature[::7], prof.altitude[::7],
                                  {s: v[::7] for s, v in prof.vmr.items()})
    d = dnu / factor
    lo, hi = 700.0, 700.0 + (n_ch - 1) * dnu
    pad = np.ceil(16.0 / d) * d
    kw = dict(backend=ctx, apply_continuum=False, high_res_factor=factor)
    snd = pkg.Sounder.make(lo, hi, dnu, opd_max=2.0, fwhm_gauss=0.5)
    mono = pkg.Sounder.make(lo - pad, hi + pad, d, opd_max=2.0, fwhm_gauss=0.5)
    _, R, BT = pkg.forward_model(prof, lists, sounder=snd, precision="fp64", **kw)
    nu, I, _ = pkg.forward_model(prof, lists, sounder=mono, precision="fp64", backend=ctx, apply_continuum=False,
                                 high_res_factor=1, with_ils=False)
    _, taps = pkg.ils_kernel(d, 2.0, 0.5, backend=ctx)
    at = len(taps) // 2 + factor * np.arange(n_ch)
    ref = pkg.apply_ils(nu, I, None, taps, backend=ctx)[at]
    assert R.shape == (n_ch,) and np.max(np.abs(R / ref - 1.0)) <= 1e-12
    spec = pkg.StateVectorSpec(len(prof.pressure), [pkg.CO2], include_emissivity=False)
    K = pkg.analytic_jacobian(prof, lists, spec, sounder=snd, observable="radiance", **kw).K
    D = pkg.analytic_jacobian(prof, lists, spec, sounder=mono, observable="radiance", backend=ctx,
                              apply_continuum=False, high_res_factor=1, with_ils=False).K
    for x in range(0, spec.n, 5):
        ref = pkg.apply_ils(nu, D[:, x], None, taps, backend=ctx)[at]
        most = pkg.apply_ils(nu, np.abs(D[:, x]), None, np.abs(taps), backend=ctx)[at]
        assert np.all(np.abs(K[:, x] - ref) <= 4.9e-5 * most + 1e-30), x
