"""A batch whose buffers do not fit beside what the context's other paths hold runs in passes:
with 9 GB left on the device, an FP64 and a mixed batch and then a batch of Jacobians (150
scenes: 11 GB at once) all succeed, and equal single scenes bit for bit."""
import numpy as np
import pytest
import torch

from conftest import load_package

pytestmark = pytest.mark.gpu


def test_paths_share_a_small_device():
    pkg = load_package()
    ctx = pkg.B200Context()
    lists = {2: pkg.synthetic.synthetic_linelist(5000, 2, 1000, 645.0, 700.0)}
    full = pkg.afgl_atmosphere("us_standard")
    n = 150
    profs = [pkg.AtmosphericProfile(full.pressure, full.temperature + 0.01 * k, full.altitude, full.vmr) for k in range(n)]
    snd = pkg.Sounder.make(645.0, 700.0, 0.25, opd_max=2.0, fwhm_gauss=0.5)
    kw = dict(sounder=snd, backend=ctx, internal_dnu=0.0025)
    spec = pkg.StateVectorSpec(len(full.pressure), [pkg.CO2], include_emissivity=False)
    torch.cuda.empty_cache()
    held = torch.empty(max(torch.cuda.mem_get_info()[0] - (9 << 30), 0), dtype=torch.uint8, device="cuda")
    try:
        _, _, b64 = pkg.forward_model_batch(profs, lists, precision="fp64", **kw)
        _, _, b32 = pkg.forward_model_batch(profs, lists, precision="mixed", **kw)
        _, K, y = pkg.analytic_jacobian_batch(profs, lists, spec, **kw)
    finally:
        del held
        torch.cuda.empty_cache()
    assert np.max(np.abs(b64 - b32)) < 1e-3
    for k in (0, n - 1):
        _, K1, y1 = pkg.analytic_jacobian_batch(profs[k:k + 1], lists, spec, **kw)
        assert np.array_equal(K[k], K1[0]) and np.array_equal(y[k], y1[0])
    ctx.close()
