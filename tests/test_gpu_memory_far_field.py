"""Batches of six species with 3 GB left on the device, where the far field's node values (as many
bytes as the optical depths) and the lines' index decide whether a pass fits: 200 mixed scenes (3.4
GB at once) and 120 Jacobians of the surface terms (6 GB) run in passes, and equal single scenes
bit for bit."""
import numpy as np
import pytest
import torch

from conftest import load_package

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["mixed", "fp64", "jacobian"])
def test_six_species_on_a_small_device(kind):
    pkg = load_package()
    ctx = pkg.B200Context()
    lists = {s: pkg.synthetic.synthetic_linelist(200, s, 500 + s, 645.0, 700.0) for s in pkg.synthetic.SPECIES6}
    full = pkg.afgl_atmosphere("us_standard")
    vmr = {s: full.vmr.get(s, np.full(len(full.pressure), 1e-7)) for s in lists}
    n = 120 if kind == "jacobian" else 200
    profs = [pkg.AtmosphericProfile(full.pressure, full.temperature + 0.01 * k, full.altitude, vmr) for k in range(n)]
    snd = pkg.Sounder.make(645.0, 700.0, 0.25, opd_max=2.0, fwhm_gauss=0.5)
    kw = dict(sounder=snd, backend=ctx, internal_dnu=0.0025)
    spec = pkg.StateVectorSpec(len(full.pressure), [], include_temperature=False)

    def run(p):
        if kind == "jacobian":
            return pkg.analytic_jacobian_batch(p, lists, spec, **kw)[1:]
        return pkg.forward_model_batch(p, lists, precision=kind, **kw)[1:]

    torch.cuda.empty_cache()
    held = torch.empty(max(torch.cuda.mem_get_info()[0] - (3 << 30), 0), dtype=torch.uint8, device="cuda")
    try:
        got = run(profs)
    finally:
        del held
        torch.cuda.empty_cache()
    for k in (0, n // 2, n - 1):
        assert all(np.array_equal(a[k], b[0]) for a, b in zip(got, run(profs[k:k + 1])))
    ctx.close()
