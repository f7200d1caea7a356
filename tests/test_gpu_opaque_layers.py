"""schwarzschild_rte with opaque layers, up to an infinite optical depth, in layer runs and in one
run (from 151,552 points), against the FP64 oracle with the tolerance of the other radiative
transfers (1e-12)."""
import numpy as np
import pytest

from conftest import load_package

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("depth", [1e16, 1e17, 1e18, 1e300, np.inf])
@pytest.mark.parametrize("src,eps", [("cim", 1.0), ("cim", 0.9), ("toon", 1.0), ("toon", 0.9)])
def test_opaque_layers(oracle, src, eps, depth):
    pkg = load_package()
    ctx = pkg.B200Context()
    for n, L, opaque in ((300, 9, (0,)), (300, 9, (4, 5)), (300, 9, (8,)), (300, 1, (0,)), (151552, 3, (1,))):
        g = 700.0 + 0.0025 * np.arange(n)
        tau = np.random.default_rng(L).uniform(0.0, 0.8, (n, L))
        tau[n // 2:, list(opaque)] = depth
        T_lev = np.linspace(290.0, 215.0, L + 1)
        kw = dict(mu=0.8, source_function=src, T_ave=0.5 * (T_lev[:-1] + T_lev[1:]) + 0.3 if src == "cim" else None)
        got = pkg.schwarzschild_rte(g, tau, T_lev, 292.0, eps_sfc=eps, backend=ctx, **kw)
        ref = oracle.rte(g, np.ascontiguousarray(tau.T), T_lev, 292.0, eps=eps, **kw)
        assert np.all(np.abs(got - ref) <= 1e-12 * ref), (n, L, opaque)
    ctx.close()
