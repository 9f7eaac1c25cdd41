"""The fixed-point FP64 sweep (the default FP64 path) at the edges of its range, against the FP64-pipe
sweep (selected by an explicit launch shape)."""
import numpy as np
import pytest

from conftest import relerr

pytestmark = pytest.mark.gpu

EPS = 0.02
FP64 = {"i_per_thread": 1}


def _system(n, seed):
    rng = np.random.default_rng(seed)
    x = rng.uniform(-1, 1, (n, 3))
    v = rng.normal(0, 0.3, (n, 3))
    m = rng.uniform(0.5, 1.5, n) / n
    x[0] = rng.normal(0, 0.05, 3)
    v[0] = 0.1 * rng.normal(size=3)
    m[0] = 0.02
    return x, v, m


def _run(pn, x, v, m, ic2, **kw):
    with pn.Context(x.shape[0], eps=EPS, inv_c2=ic2, **kw) as c:
        c.set_state(x, v, m)
        return c.force(), np.array(c.energy())


@pytest.mark.parametrize("n", [385, 1026, 4099])
def test_velocity_unit_of_every_other_tile(pn, n):
    """Tiles of slow and fast stars in turn: a CTA of fast rows rescales every other tile in its stage, which
    the next tile but one is then copied to.  The sums are the same each time, and within the 1e-12 of
    every FP64 path here of those of the FP64-pipe sweep."""
    x, v, m = _system(n, n)
    slow = (np.arange(n - 1) // 128) % 2 == 1
    v[1:][slow] *= 1e-3
    a, e = _run(pn, x, v, m, 1.0)
    b, f = _run(pn, x, v, m, 1.0, **FP64)
    assert relerr(a, b).max() <= 1e-12
    assert np.abs(e - f).max() <= 1e-12 * np.abs(f).max()
    for _ in range(20):
        again, e2 = _run(pn, x, v, m, 1.0)
        assert np.array_equal(a, again) and np.array_equal(e, e2)
