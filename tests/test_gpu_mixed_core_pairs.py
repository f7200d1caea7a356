"""Points of a line's core where the FP32 quotient of the core is singular (IRS_MIXED): m = x^2 +
y^2 = 0 with the centre on a grid point and y lost, and q = 0 where x^2 rounds to 3/2 and y^2 is
lost beside it.  The points 32 steps away, which share a reciprocal with them, carry the peaks of
two other lines.  Against the FP64 sum of the same call, with the tolerance of the other cross
sections of this path (2e-5 of the peak)."""
import numpy as np
import pytest

from conftest import load_package

pytestmark = pytest.mark.gpu

F = np.float32
STEP, N, LO = 2.0 ** -9, 4096, 696.0  # every position below is exact in FP32


@pytest.fixture(scope="module")
def pkg():
    return load_package()


@pytest.fixture(scope="module")
def ctx(pkg):
    c = pkg.B200Context()
    yield c
    c.close()


def lines(pkg, at):
    """Three lines, `at` points from the grid's first and 32 points on either side of that."""
    ll = pkg.synthetic.synthetic_linelist(3, 2, 71, 700.0, 701.0).lines.copy()
    ll["wavenumber"] = LO + STEP * (at + np.array([-32.0, 0.0, 32.0]))
    ll["intensity"] = 1e-20
    ll["lower_energy"] = 0.0
    ll["pressure_shift"] = 0.0
    ll["air_broad"] = 0.07
    ll["temp_depend"] = 0.7
    return pkg.HITRANLinelist(ll)


def check(pkg, ctx, ll, T, p):
    grid = LO + np.arange(N) * STEP
    ref = pkg.compute_voigt_cross_sections(grid, ll, T, p, backend=ctx, precision="fp64")
    got = pkg.compute_voigt_cross_sections(grid, ll, T, p, backend=ctx, precision="mixed")
    bad = np.flatnonzero(~(np.abs(got - ref) <= 2e-5 * ref.max()))
    assert bad.size == 0, (bad, got[bad], ref[bad])


@pytest.mark.parametrize("at", [2048, 2048 + 33, 2048 + 70, 2048 + 127])  # each row of a leaf
@pytest.mark.parametrize("p", [0.0, 1e-24, 1e-20, 1e-12])
def test_centre_on_a_point(pkg, ctx, at, p):
    check(pkg, ctx, lines(pkg, at), 250.0, p)


def singular_temperature(nu, d):
    """A temperature at which the quotient's q, in FP32 as the kernel forms it, is 0 at d steps
    from a CO2 line at nu of vanishing pressure; None where no float of the line's width gives
    x^2 = 3/2."""
    gd1 = nu * 3.58126e-7 / np.sqrt(44.010)  # Doppler width over sqrt(T)
    T0 = (np.sqrt(np.log(2.0)) * STEP * d / (gd1 * np.sqrt(1.5))) ** 2
    for k in range(-20, 21):
        T = T0 * (1.0 + 2e-8 * k)
        fx = F(np.sqrt(np.log(2.0)) / (gd1 * np.sqrt(T)) * STEP)
        X = F(F(d) * F(d)) * F(fx * fx)
        if F(float(X) * float(X) + float(F(2.25 - 3.0 * float(X)))) == 0.0:
            return T
    return None


@pytest.mark.parametrize("row", [0, 1, 2, 3])
def test_zero_of_the_denominator(pkg, ctx, row):
    hits = 0
    for j in range(100, 156):  # centres 100/256 to 155/256 of a step past a point
        at, d = 2048 + 32 * row + 7 + j / 256, j / 256
        T = singular_temperature(LO + STEP * at, d)
        if T is None:
            continue
        hits += 1
        assert 150.0 < T < 500.0
        for p in (0.0, 1e-8, 1e-7):
            check(pkg, ctx, lines(pkg, at), T, p)
    assert hits >= 10
