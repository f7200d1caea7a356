"""The launches that a forward call reports (irs_stage_times) are the kernels that it launches.
With the ILS at hand and one group of layers: the grid, two passes of line parameters, the line
sum, the radiative transfer (FP64: its layers' constants first) and the channels."""
import numpy as np
import pytest

from conftest import load_package

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,method,line_sum", [
    ("fp64", "FullFaddeeva", ["tree64_far", "tree64_leaf"]), ("fp64", "PseudoVoigt", ["linesum_f64"]),
    ("mixed", "FullFaddeeva", ["cell_fill", "fw_tree", "fw_leaf"]), ("mixed", "PseudoVoigt", ["linesum_mixed"]),
    ("mixed_direct", "FullFaddeeva", ["linesum_mixed"])])
def test_forward_launches(precision, method, line_sum):
    pkg = load_package()
    ctx = pkg.B200Context()
    lists = {2: pkg.synthetic.synthetic_linelist(300, 2, 84, 690.0, 720.0)}
    snd = pkg.Sounder.make(700.0, 705.0, 0.25, opd_max=2.0, fwhm_gauss=0.5)
    want = ["grid_values", "lp_keep", "lp_write", *line_sum, *(["rte_layers"] if precision == "fp64" else []), "rte", "ils"]
    for warm in (False, True):
        pkg.forward_model(pkg.afgl_atmosphere("us_standard"), lists, sounder=snd, backend=ctx, precision=precision,
                          method=pkg.VoigtMethod[method], internal_dnu=0.0025)
        assert not warm or int(ctx.stage_times().launches) == len(want), want
    ctx.close()
