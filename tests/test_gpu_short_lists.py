"""FP64 cross sections of lists on either side of the rule that sums short ones line by line (32
lines; 96 on grids of up to 512 points), uniform grids and not, against the FP64 oracle with the
tolerance of the other FP64 cross sections (1e-12 of the peak)."""
import numpy as np
import pytest

from conftest import load_package

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_lines,n", [(1, 1), (32, 3000), (33, 3000), (32, 513), (96, 513), (96, 512), (97, 512), (97, 2)])
@pytest.mark.parametrize("method", ["FullFaddeeva", "Weideman", "PseudoVoigt"])
def test_short_lists(oracle, n_lines, n, method):
    pkg = load_package()
    ctx = pkg.B200Context()
    ll = pkg.synthetic.synthetic_linelist(n_lines, 2, 95, 660.0, 664.0)
    grid = 660.0 + np.arange(n) * 0.0025
    for g in (grid, grid + 2e-4 * np.sin(np.arange(n))):
        got = pkg.compute_voigt_cross_sections(g, ll, 250.0, 0.1, backend=ctx, method=pkg.VoigtMethod[method])
        ref = oracle.voigt_xsec(ll.lines, g, 250.0, 0.1, method=method)
        assert ref.max() > 0.0 and np.max(np.abs(got - ref)) <= 1e-12 * ref.max()
    ctx.close()
