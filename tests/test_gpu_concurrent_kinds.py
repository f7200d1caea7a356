"""Contexts on threads of one device whose calls launch the same kernels with different amounts of
shared memory (state vectors of different lengths, numbers of layers and of retrieved species): every
call succeeds and equals the same call made alone."""
import threading

import numpy as np
import pytest

from conftest import load_package

pytestmark = pytest.mark.gpu


def profile(pkg, n_lev):
    full = pkg.afgl_atmosphere("us_standard")
    p = np.geomspace(1000.0, 20.0, n_lev)
    at = lambda v: np.interp(np.log(p[::-1]), np.log(full.pressure[::-1]), v[::-1])[::-1]
    return pkg.AtmosphericProfile(p, at(full.temperature), at(full.altitude), {s: at(full.vmr[s]) for s in (1, 2, 3, 4)})


class Repeat:
    """The library with its batch calls made n times in a row, until one fails: Python's share
    of a call would keep the threads' calls apart."""

    def __init__(self, lib, n):
        self.lib, self.n = lib, n

    def __getattr__(self, name):
        f = getattr(self.lib, name)
        if "_batch" not in name:
            return f
        return lambda *a: next((rc for rc in (f(*a) for _ in range(self.n)) if rc), 0)


def test_threads_with_different_shared_memory():
    pkg = load_package()
    lists = {s: pkg.synthetic.synthetic_linelist(2, s, 90 + s, 700.0, 702.0) for s in (1, 2, 3, 4)}
    snd = pkg.Sounder.make(700.0, 701.0, 0.25, opd_max=2.0, fwhm_gauss=0.5)
    kw = dict(sounder=snd, with_ils=False, internal_dnu=None, high_res_factor=1, apply_continuum=False)

    def jacobian(n_lev, retrieved):
        prof, spec = profile(pkg, n_lev), pkg.StateVectorSpec(n_lev, retrieved)
        return lambda c: pkg.analytic_jacobian_batch([prof], lists, spec, backend=c, **kw)[1]

    def pullback(n_lev):
        prof, spec = profile(pkg, n_lev), pkg.StateVectorSpec(n_lev, [1, 2, 3, 4])
        return lambda c: pkg.vjp_batch([prof], lists, spec, np.ones(5), backend=c, **kw)[1]

    def forward(n_lev):
        prof = profile(pkg, n_lev)
        return lambda c: pkg.forward_model(prof, lists, backend=c, precision="mixed", **kw)[2]

    # per group the first is the one that the others' smaller limit would refuse
    calls = [jacobian(2, [1, 2, 3, 4]), *[jacobian(2, [2])] * 3, pullback(1150), *[pullback(900)] * 3,
             forward(1000), *[forward(760)] * 3]
    ctxs = [pkg.B200Context() for _ in calls]
    alone = [f(c) for f, c in zip(calls, ctxs)]
    faults = []

    def work(f, c, ref, n):
        c.lib = Repeat(c.lib, n)
        try:
            got = f(c)
            if not np.allclose(got, ref, rtol=1e-9, atol=1e-12 * np.max(np.abs(ref))):  # the pullback sums by atomics
                faults.append("differs from the call made alone")
        except pkg.IRSError as e:
            faults.append(str(e))

    for g, n in ((0, 10000), (4, 100), (8, 2000)):
        th = [threading.Thread(target=work, args=(calls[k], ctxs[k], alone[k], n)) for k in range(g, g + 4)]
        for t in th:
            t.start()
        for t in th:
            t.join()
    for c in ctxs:
        c.close()
    assert not faults, faults
