"""The radiative transfer with a point's layers cut into runs (grids under 151,552 points) and
in one run (longer grids): fewer layers than runs, uneven runs and points at the edges of a
block, for both source functions and a reflecting surface.

Tolerances.  FP64 against the oracle: the layer runs reorder some tens of roundings, 1e-12.
Mixed against FP64: an FP32 layer's optical depth is within 1e-6 of itself, so a transmittance
e^-t within t e^-t 1e-6 < 4e-7, dT = dB/B T / x with x = c2 nu / T > 3 below 4e-5 K a layer;
2e-4 K for up to five layers."""
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


@pytest.mark.parametrize("src", ["toon", "cim"])
@pytest.mark.parametrize("n,L", [(65, 1), (63, 2), (64, 3), (129, 4), (300, 5), (1, 7), (151551, 3), (151552, 3), (152001, 9)])
def test_fp64_runs(pkg, ctx, oracle, src, n, L):
    rng = np.random.default_rng(n + L)
    g = 700.0 + 0.0025 * np.arange(n)
    tau = rng.uniform(0.0, 0.8, (n, L)) * np.linspace(1.0, 0.1, L)[None]
    tau[: n // 8] = 1e-7
    T_lev = np.linspace(290.0, 215.0, L + 1)
    T_ave = 0.5 * (T_lev[:-1] + T_lev[1:]) + 0.3 if src == "cim" else None
    for eps in (1.0, 0.9):
        kw = dict(mu=0.8, source_function=src, T_ave=T_ave)
        got = pkg.schwarzschild_rte(g, tau, T_lev, 292.0, eps_sfc=eps, backend=ctx, **kw)
        ref = oracle.rte(g, np.ascontiguousarray(tau.T), T_lev, 292.0, eps=eps, **kw)
        assert np.max(np.abs(got - ref) / ref) < 1e-12


@pytest.mark.parametrize("src", ["toon", "cim"])
@pytest.mark.parametrize("n_lev,width", [(2, 20.0), (3, 20.0), (4, 20.0), (6, 20.0), (4, 400.0)])
def test_mixed_runs(pkg, ctx, src, n_lev, width):
    full = pkg.afgl_atmosphere("us_standard")
    k = np.linspace(0, 20, n_lev).astype(int)
    prof = pkg.AtmosphericProfile(full.pressure[k], full.temperature[k], full.altitude[k],
                                  {s: v[k] for s, v in full.vmr.items()})
    lists = {2: pkg.synthetic.synthetic_linelist(800, 2, 61, 780.0, 1250.0),
             1: pkg.synthetic.synthetic_linelist(800, 1, 62, 780.0, 1250.0)}
    snd = pkg.Sounder.make(800.0, 800.0 + width, 0.25, opd_max=2.0, fwhm_gauss=0.5)
    for eps in (1.0, 0.9):
        bt = [pkg.forward_model(prof, lists, sounder=snd, backend=ctx, internal_dnu=0.0025, precision=p, eps_sfc=eps,
                                source_function=src)[2] for p in ("fp64", "mixed")]
        assert np.max(np.abs(bt[1] - bt[0])) < 2e-4
