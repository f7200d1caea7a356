"""The Jacobian's line sum with an unbroadened line centred on a grid point, where d^2 + b^2 is 0:
the points 32 steps away, which share a reciprocal with it, carry the peaks of two other lines.
Against the FP64 oracle with the tolerance of tests/test_gpu_jacobian.py (2e-4 of each column
block's largest entry)."""
import numpy as np
import pytest

from conftest import load_package
from test_gpu_jacobian import check_vs_oracle, mk, profile

pytestmark = pytest.mark.gpu

# every position below is exact in FP32, and 32 steps are past |x| = 122, the core's reach
STEP, LO, N = 2.0 ** -8, 699.0, 1024


@pytest.mark.parametrize("at", [512, 512 + 45, 512 + 70, 512 + 127])  # each row of a leaf
@pytest.mark.parametrize("species,line_mixing", [(2, False), (2, True), (3, False)])
def test_unbroadened_line_on_a_point(oracle, orc_mod, at, species, line_mixing):
    pkg = load_package()
    ctx = pkg.B200Context()
    nu = [LO + STEP * (at + k) for k in (-32, 0, 32)]
    ll = {species: mk(orc_mod, species, [(nu[0], 1e-22, 0.07, 0.08, 250.0, 0.75, 0.0),
                                         (nu[1], 1e-22, 0.0, 0.0, 250.0, 0.75, 0.0),
                                         (nu[2], 1e-22, 0.07, 0.08, 250.0, 0.75, 0.0)])}
    prof = profile(pkg, 4, lambda p: {species: 4.0e-4 * p / 1000.0})
    prof.pressure = prof.pressure * 1e-2  # narrow peaks
    spec = pkg.StateVectorSpec(4, [species])
    y0 = {2: np.array([0.01, -0.02, 0.015])} if line_mixing else None
    check_vs_oracle(pkg, ctx, oracle, orc_mod, prof, ll, spec,
                    dict(nu_min=LO, nu_max=LO + (N - 1) * STEP, dnu=STEP, opd_max=2.0, fwhm_gauss=0.5),
                    dict(apply_continuum=False, with_ils=False, high_res_factor=1), y0=y0)
    ctx.close()
