"""An infinite cutoff is an error (the grids' layouts are sized by it: no call with one can end)."""
import numpy as np
import pytest

from conftest import load_package

pytestmark = pytest.mark.gpu


def test_infinite_cutoff_is_refused():
    pkg = load_package()
    ctx = pkg.B200Context()
    ll = pkg.synthetic.synthetic_linelist(10, 2, 85, 699.0, 702.0)
    prof = pkg.afgl_atmosphere("us_standard")
    snd = pkg.Sounder.make(700.0, 701.0, 0.25, opd_max=2.0, fwhm_gauss=0.5)
    kw = dict(sounder=snd, backend=ctx, internal_dnu=0.0025, cutoff=np.inf)
    for precision in ("fp64", "mixed"):
        with pytest.raises(pkg.IRSError, match="finite"):
            pkg.compute_voigt_cross_sections(700.0 + np.arange(100) * 0.01, ll, 250.0, 0.3, backend=ctx, precision=precision,
                                             cutoff=np.inf)
        with pytest.raises(pkg.IRSError, match="finite"):
            pkg.forward_model(prof, {2: ll}, precision=precision, **kw)
    spec = pkg.StateVectorSpec(len(prof.pressure), [2])
    with pytest.raises(pkg.IRSError, match="finite"):
        pkg.analytic_jacobian(prof, {2: ll}, spec, **kw)
    ctx.close()
