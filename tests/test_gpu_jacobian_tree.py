"""The Jacobian's line sum at the edges of its blocks (leaves of 128 points, strips of
4096), for every kind of segment (value and d/dT alone; with d/dp; with d/dv of water; with
VP_Y), narrow cutoffs and extreme cores, against the FP64 oracle's analytic Jacobian.

Tolerance: as tests/test_gpu_jacobian.py, 2e-4 of each column block's largest entry (FP32
sums whose interpolated part is within 1.6e-8 of a line's wing)."""
import numpy as np
import pytest

from conftest import load_package
from test_gpu_jacobian import check_vs_oracle, profile

pytestmark = pytest.mark.gpu

DNU = 0.0025


@pytest.fixture(scope="module")
def pkg():
    return load_package()


@pytest.fixture(scope="module")
def ctx(pkg):
    c = pkg.B200Context()
    yield c
    c.close()


def lists(pkg, n, lo=675.0, hi=735.0):
    return {s: pkg.synthetic.synthetic_linelist(n, s, 60 + s, lo, hi).lines for s in (1, 2, 3)}


def atm(pkg, nlev=5):
    return profile(pkg, nlev, lambda p: {1: 8e-3 * p / 1000.0, 2: np.full(len(p), 4.0e-4), 3: 2e-6 * 500.0 / p})


def snd(n, lo=700.0, dnu=DNU):
    return dict(nu_min=lo, nu_max=lo + (n - 1) * dnu, dnu=dnu, opd_max=2.0, fwhm_gauss=0.5)


@pytest.mark.parametrize("n", [1, 127, 129, 4096, 4097, 4225])
@pytest.mark.parametrize("retrieved", [[], [2], [1, 3]])
def test_sizes_and_kinds(pkg, ctx, oracle, orc_mod, n, retrieved):
    prof = atm(pkg)
    spec = pkg.StateVectorSpec(len(prof.pressure), retrieved)
    check_vs_oracle(pkg, ctx, oracle, orc_mod, prof, lists(pkg, 150), spec, snd(n),
                    dict(apply_continuum=False, with_ils=False, high_res_factor=1))


@pytest.mark.parametrize("retrieved", [[3], [2, 1]])
def test_line_mixing_kinds(pkg, ctx, oracle, orc_mod, retrieved):
    prof = atm(pkg)
    ll = lists(pkg, 200)
    spec = pkg.StateVectorSpec(len(prof.pressure), retrieved)
    check_vs_oracle(pkg, ctx, oracle, orc_mod, prof, ll, spec, snd(2100),
                    dict(apply_continuum=False, with_ils=False, high_res_factor=1),
                    y0={2: pkg.synthetic.vpy_y0(len(ll[2]), seed=61)})


# cutoffs narrower than a leaf, a strip, and past the strip; cores from 5 Doppler widths to
# wider than the cutoff
@pytest.mark.parametrize("cutoff,x_far", [(0.2, 122.0), (3.0, 122.0), (6.0, 5.0), (2.0, 1e5)])
def test_windows(pkg, ctx, oracle, orc_mod, cutoff, x_far):
    prof = atm(pkg)
    spec = pkg.StateVectorSpec(len(prof.pressure), [1])
    check_vs_oracle(pkg, ctx, oracle, orc_mod, prof, lists(pkg, 150), spec, snd(1500),
                    dict(apply_continuum=False, with_ils=False, high_res_factor=1, cutoff=cutoff, x_far=x_far))


def test_node_buffer_groups(pkg, monkeypatch):
    """The far field's node values in groups of profile-layers that fit the buffer: K does not
    depend on the groups; without room for one profile-layer every line is summed at the
    points, and K agrees to FP32 rounding (1e-5 of each row's largest entry)."""
    ll = {s: pkg.HITRANLinelist(v) for s, v in lists(pkg, 150).items()}
    prof = atm(pkg)
    spec = pkg.StateVectorSpec(len(prof.pressure), [1, 3])
    s = pkg.Sounder.make(**snd(4300))
    K = []
    cell = 4 * 16 * 4 + 16
    for limit in (None, 3 * 64 * cell + 100, 1000):  # all layers, one layer at a time, none
        if limit:
            monkeypatch.setenv("IRS_STRIP_BUFFER_BYTES", str(limit))
        c = pkg.B200Context()
        K.append(pkg.analytic_jacobian(prof, ll, spec, sounder=s, backend=c, apply_continuum=False, with_ils=False,
                                       high_res_factor=1).K)
        c.close()
    assert np.array_equal(K[0], K[1])
    assert np.all(np.abs(K[2] - K[0]) <= 1e-5 * np.max(np.abs(K[0]), axis=0))


@pytest.mark.parametrize("lo", [20.0, 700.0, 2300.0])  # radfn's three branches (c2 nu/T below 0.01 .. above 10)
@pytest.mark.parametrize("source_function,eps", [("cim", 1.0), ("cim", 0.9), ("toon", 1.0), ("toon", 0.9)])
def test_radiative_transfer_terms(pkg, ctx, oracle, orc_mod, lo, source_function, eps):
    """The continua's and the source functions' derivatives (both sources, reflecting surface)
    with thin and thick layers, at wavenumbers where each branch of the terms is taken."""
    prof = atm(pkg, 7)
    ll = {s: pkg.synthetic.synthetic_linelist(30, s, 80 + s, max(lo - 8.0, 1.0), lo + 16.0).lines for s in (1, 2)}
    spec = pkg.StateVectorSpec(len(prof.pressure), [1, 2])
    check_vs_oracle(pkg, ctx, oracle, orc_mod, prof, ll, spec, snd(300, lo, 0.02),
                    dict(apply_continuum=True, continua=("h2o", "co2"), with_ils=False, high_res_factor=1,
                         source_function=source_function), eps=eps)
