"""irs_jacobian_batch_rows against irs_jacobian_batch: the same K with its axes exchanged, bit for
bit, over sizes below, at and above the page-locked halves it is brought down through (2^18
values) and with channels on and off the internal grid's nodes."""
import ctypes as C

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


@pytest.mark.parametrize("n_prof,n_ch,kw", [(1, 1, dict(high_res_factor=20)), (3, 1024, dict(high_res_factor=20)),
                                            (4, 1024, dict(high_res_factor=20)), (4, 3301, dict(high_res_factor=20)),
                                            (2, 1500, dict(internal_dnu=0.03))])
def test_layouts_agree(pkg, ctx, n_prof, n_ch, kw):
    lists = {2: pkg.synthetic.synthetic_linelist(60, 2, 71, 690.0, 740.0)}
    full = pkg.afgl_atmosphere("tropical")
    profs = [pkg.AtmosphericProfile(full.pressure, full.temperature + k, full.altitude, full.vmr) for k in range(n_prof)]
    spec = pkg.StateVectorSpec(len(full.pressure), [pkg.CO2])
    snd = pkg.Sounder.make(700.0, 700.0 + 0.25 * (n_ch - 1), 0.25, opd_max=2.0, fwhm_gauss=0.5)
    _, K, y = pkg.analytic_jacobian_batch(profs, lists, spec, sounder=snd, backend=ctx, apply_continuum=False, **kw)
    assert K.shape == (n_prof, n_ch, spec.n) and K.flags.c_contiguous
    o = pkg.fm_options(line_mixing=None, dptmn=0.0, apply_continuum=False, **kw)
    cs, keep = pkg.estimation._c_spec(spec, spec.log_vmr, True, "bt")
    batch = pkg._ProfileBatch(profs, [None] * n_prof, [1.0] * n_prof, [1.0] * n_prof)
    Kc, yc = np.empty((n_prof, spec.n, n_ch)), np.empty((n_prof, n_ch))
    pkg.check(ctx.lib.irs_jacobian_batch(ctx.h, batch.arr, n_prof, C.byref(snd.c_struct()), C.byref(o), C.byref(cs),
                                         pkg.dptr(Kc), pkg.dptr(yc)))
    assert np.array_equal(K, np.transpose(Kc, (0, 2, 1))) and np.array_equal(y, yc)
    assert np.abs(K).max() > 0.0
