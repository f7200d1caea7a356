"""A call that fails because the device has no memory left leaves the context usable: made again
once there is memory, it gives what a fresh context gives.  The calls are warmed up by PseudoVoigt,
which allocates everything but the block sums' own buffers, so the first of these, their constant
tables, is the allocation that fails."""
import contextlib
import ctypes as C

import numpy as np
import pytest

from conftest import load_package

pytestmark = pytest.mark.gpu


@contextlib.contextmanager
def full_device():
    """Every free byte of the current device's memory taken, down to 256-byte pieces."""
    cuda = C.CDLL("libcuda.so.1")
    held, size = [], 1 << 34
    try:
        while size >= 256:
            d = C.c_uint64()
            if cuda.cuMemAlloc_v2(C.byref(d), C.c_size_t(size)) == 0:
                held.append(d)
            else:
                size //= 2
        yield
    finally:
        for d in held:
            cuda.cuMemFree_v2(d)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_tables_after_a_failed_allocation(precision):
    pkg = load_package()
    ll = pkg.synthetic.synthetic_linelist(600, 2, 82, 640.0, 720.0)
    grid = 660.0 + np.arange(5000) * 0.0025
    call = lambda c, m: pkg.compute_voigt_cross_sections(grid, ll, 250.0, 0.3, backend=c, precision=precision, method=m)
    fresh = pkg.B200Context()
    ref = call(fresh, pkg.FullFaddeeva)
    fresh.close()
    c = pkg.B200Context()
    call(c, pkg.VoigtMethod.PseudoVoigt)
    with full_device():
        with pytest.raises(pkg.IRSError, match="allocation of"):
            call(c, pkg.FullFaddeeva)
    assert np.array_equal(call(c, pkg.FullFaddeeva), ref)
    c.close()


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_ils_after_a_failed_allocation(precision):
    """A second sounder with more taps but a shorter grid: its ILS is the allocation that fails.
    The first sounder's taps are made anew."""
    pkg = load_package()
    lists = {2: pkg.synthetic.synthetic_linelist(300, 2, 83, 700.0, 800.0)}
    prof = pkg.afgl_atmosphere("us_standard")
    snd = [pkg.Sounder.make(lo, hi, 0.25, opd_max=2.0, fwhm_gauss=0.5) for lo, hi in ((700.0, 1000.0), (750.0, 750.25))]
    c = pkg.B200Context()
    call = lambda k: pkg.forward_model(prof, lists, sounder=snd[k], backend=c, precision=precision,
                                       internal_dnu=(0.0025, 0.001)[k], apply_continuum=False)[2]
    ref = call(0)
    with full_device():
        with pytest.raises(pkg.IRSError, match=r"allocation of .* \(ils\)"):
            call(1)
    assert np.array_equal(call(0), ref)
    c.close()
