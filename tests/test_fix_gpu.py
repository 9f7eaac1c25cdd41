"""The fixed-point FP64 sweep (the default FP64 path) against the FP64-pipe sweep (selected by an
explicit launch shape) and the oracle, at tile edges and remainders, and its range check: systems
outside the fixed-point range take the general block in the same launch.

Tolerance 1e-12 per particle (normwise), as for every FP64 path here: both sweeps stay within a few
units of FP64 rounding of the sums of their terms' magnitudes, which for these systems are at most
some hundred times the accelerations."""
import numpy as np
import pytest

from conftest import relerr

pytestmark = pytest.mark.gpu

EPS = 0.02


def _system(n, seed):
    rng = np.random.default_rng(seed)
    x = rng.uniform(-1, 1, (n, 3))
    v = rng.normal(0, 0.3, (n, 3))
    m = rng.uniform(0.5, 1.5, n) / n
    x[0] = rng.normal(0, 0.05, 3)
    v[0] = 0.1 * rng.normal(size=3)
    m[0] = 0.02
    return x, v, m


def _both(pn, x, v, m, ic2, eps=EPS):
    out = []
    for kw in ({}, {"i_per_thread": 1}):
        with pn.Context(x.shape[0], eps=eps, inv_c2=ic2, dt=1e-3, **kw) as c:
            c.set_state(x, v, m)
            out.append((c.force(), np.array(c.energy()), np.array(c.steps_energy(2)), *c.get_state()))
    return out


def _same(a, b):
    assert relerr(a[0], b[0]).max() <= 1e-12
    for e, f in ((a[1], b[1]), (a[2], b[2])):
        assert np.abs(e - f).max() <= 1e-12 * np.abs(f).max()
    assert np.abs(a[3] - b[3]).max() <= 1e-12 * np.abs(b[3]).max()
    assert np.abs(a[4] - b[4]).max() <= 1e-12 * np.abs(b[4]).max()


@pytest.mark.parametrize("ic2", [0.0, 1e-6, 1.0])
@pytest.mark.parametrize("n", [2, 3, 9, 128, 129, 130, 257, 1026, 2049, 4099])
def test_matches_fp64_sweep(pn, oracle, n, ic2):
    x, v, m = _system(n, n)
    new, old = _both(pn, x, v, m, ic2)
    _same(new, old)
    if ic2 == 1.0 and n <= 1026:
        assert relerr(new[0], oracle.force(x, v, m, EPS)).max() <= 1e-12


@pytest.mark.parametrize("what", ["far", "light", "heavy", "negative"])
def test_outside_the_range(pn, what):
    n = 300
    x, v, m = _system(n, 7)
    k = 77
    if what == "far":
        x[k] = [EPS * 2.0 ** 25, 1.0, 0.0]
    elif what == "light":
        m[k] = m[0] * 2.0 ** -40
    elif what == "heavy":
        m[k] = m[0] * 2.0 ** 61
    else:
        m[k] = -m[k]
    new, old = _both(pn, x, v, m, 1e-6)
    scale = np.abs(old[0]).max(axis=1, initial=1e-300)
    assert (np.abs(new[0] - old[0]).max(axis=1) <= 1e-12 * np.maximum(scale, np.abs(old[0]).max() * 1e-3)).all()


def test_range_flag_is_cleared(pn):
    """An evaluation outside the range leaves no trace in the next one."""
    x, v, m = _system(500, 3)
    with pn.Context(500, eps=EPS) as c:
        c.set_state(x, v, m)
        a = c.force()
        w = m.copy()
        w[9] = -w[9]
        c.set_state(x, v, w)
        c.force()
        c.energy()
        c.set_state(x, v, m)
        assert np.array_equal(c.force(), a)


def test_velocity_units_of_tiles(pn):
    """One tile of stars at rest, one of fast stars, one of slow ones."""
    x, v, m = _system(400, 5)
    v[1:129] = 0.0
    v[129:257] *= 3.0
    v[257:] *= 1e-4
    new, old = _both(pn, x, v, m, 1e-2)
    _same(new, old)


def test_nonfinite_state_is_reported(pn):
    x, v, m = _system(200, 4)
    x[50, 1] = np.nan
    with pn.Context(200, eps=EPS) as c:
        c.set_state(x, v, m)
        with pytest.raises(pn.PNError) as e:
            c.force()
        assert e.value.status == -4
