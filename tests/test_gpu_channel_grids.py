"""Channel grids whose common denominator exceeds what integers in double hold: the ends are
p/q with primes q near a million and the step a hundredth of 100/10007, so the numerators pass
2^63.  Against the same sounder with its ends 1e-9 cm^-1 off, which have no rational form: the
spectra differ by 1e-9 of their slope (below 1e4 K per cm^-1 after the ILS), 1e-4 K allowed."""
import numpy as np
import pytest

from conftest import load_package

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_large_denominators(precision):
    pkg = load_package()
    ctx = pkg.B200Context()
    lists = {2: pkg.synthetic.synthetic_linelist(600, 2, 81, 1080.0, 1120.0)}
    full = pkg.afgl_atmosphere("us_standard")
    k = np.arange(0, 20, 4)
    prof = pkg.AtmosphericProfile(full.pressure[k], full.temperature[k], full.altitude[k],
                                  {s: v[k] for s, v in full.vmr.items()})
    out = []
    for e in (0.0, 1e-9):
        snd = pkg.Sounder.make(1100189551 / 999979 + e, 1101048729 / 999983 + e, 100 / 10007, opd_max=2.0, fwhm_gauss=0.5)
        kw = dict(sounder=snd, backend=ctx, internal_dnu=None, high_res_factor=100, apply_continuum=False)
        bt = pkg.forward_model(prof, lists, precision=precision, **kw)[2]
        K = pkg.analytic_jacobian(prof, lists, pkg.StateVectorSpec(len(k), [2]), **kw).K if precision == "mixed" else bt
        out.append((bt, K))
    assert len(out[0][0]) == len(out[1][0]) > 60 and np.ptp(out[1][0]) > 1.0
    assert np.max(np.abs(out[0][0] - out[1][0])) < 1e-4
    assert np.max(np.abs(out[0][1] - out[1][1])) < 1e-4 * np.max(np.abs(out[1][1]))
    ctx.close()
