"""The range check of the fixed-point FP64 sweep (pn_fix.cuh), compiled for the CPU."""
import subprocess

import numpy as np
import pytest

from test_fix_algebra import U, row  # noqa: F401

CPP = __file__.replace("test_fix_range.py", "fix_range.cpp")


@pytest.fixture(scope="module")
def inside(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("fix") / "fix_range")
    subprocess.run(["g++", "-O2", "-std=c++17", "-Wno-unknown-pragmas", "-o", exe, CPP], check=True)

    def run(m0=0.02, m=1e-3, v2=0.09, s=(0.5, 0.2, -0.1), eL=-6, ic2=0.0):
        line = " ".join("%.17g" % q for q in (m0, m, v2, *s)) + " %d %.17g\n" % (eL, ic2)
        return subprocess.run([exe], input=line, capture_output=True, text=True, check=True).stdout.strip() == "1"

    return run


def test_signs_and_values(inside):
    inf, nan = float("inf"), float("nan")
    assert inside() and inside(m=0.0) and inside(v2=0.0) and inside(s=(0.0, 0.0, 0.0))
    assert not inside(m0=-0.02) and not inside(m0=0.0) and not inside(m=-1e-3)
    for bad in (inf, -inf, nan):
        assert not inside(m0=bad) and not inside(m=bad) and not inside(v2=bad) and not inside(s=(0.5, bad, 0.1))
    assert inside(m=0.02 * 2.0 ** -31) and not inside(m=0.02 * 2.0 ** -33)
    assert inside(m=0.02 * 2.0 ** 57) and not inside(m=0.02 * 2.0 ** 60)
    assert inside(s=(2.0 ** 17.9, 0, 0)) and not inside(s=(2.0 ** 18.1, 0, 0))


def test_units_that_a_double_holds(inside):
    """The exponents of a tile's sums (the kernel's formulas) at the limits that the check lets through."""
    def largest(ok, lo, hi):  # the last k from lo on towards hi that is inside
        step = 1 if hi > lo else -1
        k = lo
        while k != hi and ok(k + step):
            k += step
        return k

    def star(e0, eL, k):  # at rest next to the BH, of the BH's mass, v^2 = 2^k
        return inside(m0=2.0 ** e0, m=2.0 ** e0, v2=2.0 ** k, s=(2.0 ** (eL - 3), 0, 0), eL=eL)

    for eL in (-60, 0, 60):
        lo = largest(lambda e: star(e, eL, -1000), 0, -1000)
        hi = largest(lambda e: star(e, eL, -1000), 0, 1000)
        for e0 in (lo, hi):
            ev = largest(lambda k: star(e0, eL, k), -1000, 1000) // 2 + 2
            for e in (ev, -200):  # the fastest star, one at rest
                for g in (-126, 67):  # exponent of a tile's sum of m Q^2: none, the heaviest
                    gn = g + e0 - 2 * eL
                    h = g + e0 - 2 * eL + 2 + 2 * e
                    units = [gn - 62, gn - eL - 60, gn + 2 - 2 - 62 + 2 * e, gn + 2 - 14 - 62 + 2 * e, gn + 2 - 14 - 62 + e]
                    units += [max(c + 2 * e0 - 3 * eL, h - lift) + 1 - 62 for c in (-126, 128) for lift in (2, 18)]
                    assert min(units) >= -1022 and max(units) <= 1023, (e0, eL, e, g, units)


def test_speeds(inside):
    for ic2 in (1.0, 0.7, 1e-6, 3.1e-6, 1e6):
        c = ic2 ** -0.5
        assert inside(v2=c * c, ic2=ic2) and inside(v2=0.0, ic2=ic2), ic2
        assert not inside(v2=9.0 * c * c, ic2=ic2), ic2
    assert inside(v2=1e20, m0=1e30, m=1e27, ic2=0.0)
    assert not inside(v2=0.09, ic2=float("inf"))


@pytest.mark.parametrize("ic2", [1.0, 1e-6])
@pytest.mark.parametrize("mode", [1, 2, 3])
def test_one_fast_star(row, inside, mode, ic2):  # noqa: F811
    """A light star at the largest speed that the check lets through, the others slow: the errors of W and Psi
    stay below 16 units of FP64 rounding (u = 2^-53) of the sum of their terms' magnitudes, and of G's and Phi's
    beside which inv_c2 weights them."""
    rng = np.random.default_rng(mode)
    n, c = 128, ic2 ** -0.5
    s = rng.normal(0, 1, (n, 3))
    v = np.clip(rng.normal(0, 1, (n, 3)) * 0.2, -0.5, 0.5)
    m = rng.uniform(0.5, 1.5, n) / n
    m[5] = 0.02 * 2.0 ** -31
    fast = max(f for f in np.arange(1.0, 6.0, 0.05) if inside(v2=(f * c) ** 2, ic2=ic2))
    v[5] = fast * c * np.array([0.6, 0.0, 0.8])
    for i in (0, 5, 60, 127):
        r = row(mode, s, v, m, i, 1e-2, 0.02)
        if mode != 2:
            assert (np.abs(r[6:9, 2]) <= 16 * U * (r[6:9, 4] + r[0:3, 4] / ic2)).all(), (i, fast)
        if mode != 1:
            assert abs(r[9, 2]) <= 16 * U * (r[9, 4] + r[3, 4] / ic2), (i, fast)
