"""The range check of the fixed-point FP64 sweep (pn_fix.cuh), compiled for the CPU."""
import subprocess

import pytest

CPP = __file__.replace("test_fix_range.py", "fix_range.cpp")


@pytest.fixture(scope="module")
def inside(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("fix") / "fix_range")
    subprocess.run(["g++", "-O2", "-std=c++17", "-Wno-unknown-pragmas", "-o", exe, CPP], check=True)

    def run(m0=0.02, m=1e-3, v2=0.09, s=(0.5, 0.2, -0.1), eL=-6):
        line = " ".join("%.17g" % q for q in (m0, m, v2, *s)) + " %d\n" % eL
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
