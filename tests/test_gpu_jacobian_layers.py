"""The Jacobian's radiative transfer where its tables of exponentials change: more layers than
it holds at a time (64), wavenumbers where 1 - exp(-c2 nu/T) cancels, a coarse internal grid
on which a block of points spans several continuum knots, the last block of a grid, both
source functions; K against the FP64 oracle's analytic Jacobian.

Tolerance: K is linear in FP32 line sums, within 2e-5 of the peak each for tau and its
derivatives; a column block is compared with its largest entry, as in test_gpu_jacobian.py:
2e-4."""
import numpy as np
import pytest

from conftest import load_package
from test_gpu_jacobian import check_vs_oracle, mk, profile

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def pkg():
    return load_package()


@pytest.fixture(scope="module")
def ctx(pkg):
    c = pkg.B200Context()
    yield c
    c.close()


@pytest.mark.parametrize("src", ["cim", "toon"])
@pytest.mark.parametrize("nlev,nu0,dnu", [(64, 699.0, 0.005), (65, 699.0, 0.005), (66, 699.0, 0.005), (140, 699.0, 0.005),
                                          (6, 30.0, 0.005), (66, 30.0, 0.05), (9, 700.0, 0.1)])
def test_layers_and_ranges(pkg, ctx, oracle, orc_mod, src, nlev, nu0, dnu):
    ll = {1: mk(orc_mod, 1, [(nu0 + 1.6, 3.0e-22, 0.09, 0.45, 200.0, 0.70, 0.005),
                             (nu0 + 3.3, 1.2e-22, 0.09, 0.45, 450.0, 0.70, 0.005)])}
    prof = profile(pkg, nlev, lambda p: {1: 0.01 * np.exp(-3.0 * (1000.0 - p) / 800.0)})
    spec = pkg.StateVectorSpec(nlev, [1])
    check_vs_oracle(pkg, ctx, oracle, orc_mod, prof, ll, spec,
                    dict(nu_min=nu0, nu_max=nu0 + 6.0, dnu=0.5, opd_max=2.0, fwhm_gauss=0.5),
                    dict(apply_continuum=True, continua=("h2o",), with_ils=True, internal_dnu=dnu, source_function=src),
                    eps=0.9)


def test_adjoint_with_a_long_state(pkg, ctx):
    """The adjoint's sums of a state near the accepted 6,144 elements lie beside the tables in
    shared memory: dx = K^T dy of irs_vjp_batch against K of irs_jacobian_batch (K rounded to
    FP32 by column, 13 channels: 1e-6 of sum |K| |dy|, 2e-5 for the FP32 channel sums)."""
    nlev = 3000
    ll = {1: pkg.synthetic.synthetic_linelist(3, 1, 5, 700.0, 704.0)}
    prof = profile(pkg, nlev, lambda p: {1: 0.01 * np.exp(-3.0 * (1000.0 - p) / 800.0)})
    spec = pkg.StateVectorSpec(nlev, [1])
    snd = pkg.Sounder.make(699.0, 705.0, 0.5, opd_max=2.0, fwhm_gauss=0.5)
    kw = dict(sounder=snd, backend=ctx, internal_dnu=0.1, T_sfcs=[290.0], eps_sfcs=[0.98])
    _, K, _ = pkg.analytic_jacobian_batch([prof], ll, spec, **kw)
    dy = np.linspace(0.5, 1.5, K.shape[1])
    _, dx = pkg.vjp_batch([prof], ll, spec, dy, **kw)
    assert np.all(np.abs(dx[0] - dy @ K[0]) <= 2.1e-5 * (dy @ np.abs(K[0])) + 1e-12)
