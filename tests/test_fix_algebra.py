"""The fixed-point pair terms of the FP64 sweep (pn_fix.cuh), compiled for the CPU.

tests/fix_pairs.cpp runs one star's row through the same functions as the GPU kernel (integer
arithmetic: the same bits for the same seeds) and through plain FP64 and long double.  The bound
of every sum is 16 units of FP64 rounding (u = 2^-53) of the sum of its terms' magnitudes: the
per-star constants (R, mu3, ...) are formed in FP64 with up to 8 u each, as in the plain sweep,
and the sums themselves stay below 4 u.  W and Psi are weighted by inv_c2 beside G and Phi.
"""
import subprocess

import numpy as np
import pytest

U = 2.0 ** -53
CPP = __file__.replace("test_fix_algebra.py", "fix_pairs.cpp")


@pytest.fixture(scope="module")
def row(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("fix") / "fix_pairs")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-Wno-unknown-pragmas", "-o", exe, CPP], check=True)

    def run(mode, s, v, m, i, eps, m0, seed_error=3e-7):
        rows = "\n".join(" ".join("%.17g" % q for q in (*s[j], *v[j], m[j])) for j in range(len(m)))
        head = "%d %d %d %.17g %.17g %.17g\n" % (mode, len(m), i, eps, m0, seed_error)
        out = subprocess.run([exe], input=head + rows, capture_output=True, text=True, check=True).stdout
        return np.array([[float(q) for q in line.split()] for line in out.splitlines()])

    return run


def _check(r, ic2, mode, tag):
    mag = r[:, 4].copy()
    mag[6:9] = mag[0:3] / ic2 + mag[6:9]
    mag[9] += mag[3] / ic2
    use = {0: [0, 1, 2], 1: range(9), 2: [3, 9], 3: range(10)}[mode]
    err = np.abs(r[:, 2]) / mag / U
    for q in use:
        assert err[q] <= 16.0, (tag, q, err)


@pytest.mark.parametrize("mode", [0, 1, 2, 3])
@pytest.mark.parametrize("n,vs,ic2,eps,masses", [
    (300, 0.4, 1.0, 0.02, 0), (129, 1.0, 1.0, 1e-3, 0), (700, 0.7, 1e-6, 6e-4, 5), (260, 0.0, 1.0, 1e-3, 0),
    (3, 0.3, 1.0, 0.5, 0), (200, 0.3, 1.0, 50.0, 0), (256, 0.3, 1e-6, 1e-6, 2)])
def test_row_sums(row, mode, n, vs, ic2, eps, masses):
    rng = np.random.default_rng(n)
    s = rng.normal(0, 1, (n, 3)) * rng.uniform(0.05, 3, (n, 1))
    s[:min(8, n // 2)] *= 10.0  # halo stars
    if n > 100:  # a close pair, coincident stars, a star next to the BH
        s[20] = s[21] + eps * rng.normal(0, 1, 3)
        s[22] = s[23]
        s[24] *= 1e-4
    s = np.clip(s, -2.0 ** 23 * eps, 2.0 ** 23 * eps)
    v = np.clip(rng.normal(0, 1, (n, 3)) * vs, -1.1, 1.1)
    m = rng.uniform(0.5, 1.5, n) / n * 10.0 ** rng.uniform(-masses, 0, n)
    if masses:
        m[5] = 0.0
    for i in sorted({0, 20 % n, 22 % n, 24 % n, n - 1}):
        _check(row(mode, s, v, m, i, eps, 0.02), ic2, mode, (n, i))


def test_seed_at_powers_of_two(row):
    """Distances whose inverse lies next to a power of two, seeds off by up to 3e-7 on either side."""
    rng = np.random.default_rng(1)
    for _ in range(60):
        p = 2.0 ** rng.integers(0, 12) * (1 + rng.normal() * 1e-7)
        u = rng.normal(0, 1, 3)
        s = np.array([[0.3, 0.2, 0.1], [0.3, 0.2, 0.1] + u / np.linalg.norm(u) * np.sqrt(max(0.0, p * p - 1.0))])
        _check(row(1, s, rng.normal(0, 0.3, (2, 3)), np.array([1e-3, 2e-3]), 0, 1.0, 0.02), 1.0, 1, p)
