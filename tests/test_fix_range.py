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
