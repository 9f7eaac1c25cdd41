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


def _device(pn, x, v, m, ic2, eps=EPS, **kw):
    torch = pytest.importorskip("torch")
    n = len(x)
    with pn.Context(n, eps=eps, inv_c2=ic2, **kw) as c:
        d = [torch.tensor(q, device="cuda") for q in (x, v, m)]
        a = torch.full((n, 3), np.nan, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        c.force_device(n, *(q.data_ptr() for q in d), a.data_ptr(), 0)
        c.sync()
        return a.cpu().numpy()


def _same(a, b, scale=1e-3):
    """Within 1e-12 of the larger of a particle's acceleration and scale times the largest one."""
    na = np.linalg.norm(b, axis=1)
    assert (np.linalg.norm(a - b, axis=1) <= 1e-12 * np.maximum(na, scale * na.max())).all()


@pytest.mark.parametrize("ic2", [0.0, 1e-6, 1e-2])
def test_negative_bh_mass(pn, ic2):
    """pn_force_device cannot look at the masses: a BH mass below zero gives the formula's value.  (With the star
    next to the BH and inv_c2 = 1, two shapes of the FP64-pipe sweep already differ by 1.2e-12.)"""
    x, v, m = _system(300, 11)
    x[7] = x[0] + 1e-3
    m[0] = -m[0]
    _same(_device(pn, x, v, m, ic2), _device(pn, x, v, m, ic2, **FP64))


@pytest.mark.parametrize("mass,length", [(-500, 0), (-340, 50), (340, -50), (480, 0), (-294, -54), (-294, 66),
                                         (-290, 0), (290, 0), (306, 66), (306, -54)])
def test_extreme_units(pn, mass, length):
    """Units far from 1 (masses and lengths times powers of two), inside the range and outside."""
    x, v, m = _system(300, 13)
    x[5] = x[0] + 1e-4
    v[1:129] *= 1e-3
    s = 2.0 ** ((mass - length) // 2)
    a, b = (_device(pn, x * 2.0 ** length, v * s, m * 2.0 ** mass, 1e-2 / s ** 2, eps=EPS * 2.0 ** length, **kw)
            for kw in ({}, FP64))
    assert np.isfinite(b).all() and np.abs(b).max() > 0
    _same(a, b)


@pytest.mark.parametrize("speed", [0.5, 3.0, 10.0, 30.0, 1e2, 1e3, 1e4, 1e5])
def test_one_fast_star(pn, speed):
    """One light star far faster than the rest, and than c: the slow rows keep their velocity sums."""
    x, v, m = _system(300, 17)
    m[40] = m[0] * 2.0 ** -31
    v[40] = speed * np.array([0.6, 0.0, 0.8])
    new, old = (_run(pn, x, v, m, 1.0, **kw) for kw in ({}, FP64))
    assert relerr(new[0], old[0]).max() <= 1e-12
    assert np.abs(new[1] - old[1]).max() <= 1e-12 * np.abs(old[1]).max()


@pytest.mark.parametrize("ic2", [0.0, 1.0])
@pytest.mark.parametrize("sep", [1e-1, 1e-2, 1e-4, 1e-6, 1e-8, 1e-10])
@pytest.mark.parametrize("n", [3, 5])
def test_close_pair_that_dominates(pn, n, sep, ic2):
    """Two stars far below the softening apart, beside a BH too light to matter, alone or with a third one far
    off: the pair's force keeps FP64's relative accuracy.  (An energy in between: one sweep serves both.)"""
    rng = np.random.default_rng(n)
    x = np.zeros((n, 3))
    x[1] = [0.25, -0.125, 0.5]
    x[2] = x[1] + sep * EPS * np.array([0.6, 0.0, 0.8])
    x[3:] = rng.uniform(-1, 1, (n - 3, 3)) * 1e3
    v = rng.normal(0, 0.3, (n, 3))
    m = np.full(n, 1.0)
    m[0] = 2.0 ** -50
    out = []
    for kw in ({}, FP64):
        with pn.Context(n, eps=EPS, inv_c2=ic2, dt=1e-3, **kw) as c:
            c.set_state(x, v, m)
            a = c.force()
            e = np.array(c.steps_energy(1))
            out.append((a, e, c.get_state()[1] - v))
    new, old = out
    assert relerr(new[0][1:], old[0][1:]).max() <= 1e-14
    assert np.abs(new[1] - old[1]).max() <= 1e-12 * np.abs(old[1]).max()


@pytest.mark.parametrize("ic2", [0.0, 1.0])
@pytest.mark.parametrize("n", [130, 300, 1026, 2500, 9001])
def test_close_pairs_among_others(pn, n, ic2):
    """Four heavy pairs, each 1e-7 eps wide, at the ends and in the middle of the rows, among light stars."""
    x, v, m = _system(n, n)
    m[:] = 1e-12
    corners = np.array([[1.0, 1.0, 1.0], [1.0, -1.0, -1.0], [-1.0, 1.0, -1.0], [-1.0, -1.0, 1.0]])
    rng = np.random.default_rng(n)
    for k, (i, j) in enumerate([(1, 2), (5, 129), (n // 2, n - 2), (n // 3, n - 1)]):
        x[i] = corners[k]
        x[j] = x[i] + 1e-7 * EPS * rng.normal(size=3)
        m[[i, j]] = 1.0
    new, old = (_run(pn, x, v, m, ic2, **kw) for kw in ({}, FP64))
    assert relerr(new[0], old[0]).max() <= 1e-12


@pytest.mark.parametrize("n", [2, 9, 17, 129, 1026, 4099, 9001])
def test_general_block_of_any_size(pn, n):
    """A system outside the range, its FP64 items shared out among the CTAs: the sums of the FP64-pipe sweep,
    the same each time, in force, energy and step."""
    x, v, m = _system(n, n)
    m[n // 2 or 1] = m[0] * 2.0 ** -40
    out = []
    for kw in ({}, {}, FP64):
        with pn.Context(n, eps=EPS, inv_c2=1e-2, dt=1e-3, **kw) as c:
            c.set_state(x, v, m)
            a, again = c.force(), c.force()
            assert np.array_equal(a, again)
            out.append((a, np.array(c.energy()), np.array(c.steps_energy(2)), *c.get_state()))
    for p, q in zip(out[0], out[1]):
        assert np.array_equal(p, q)
    assert relerr(out[0][0], out[2][0]).max() <= 1e-12
    for p, q in zip(out[0][1:], out[2][1:]):
        assert np.abs(p - q).max() <= 1e-12 * np.abs(q).max()


@pytest.mark.parametrize("kw,variant", [
    ({}, 6), (FP64, 1), ({"eps": 1e-25}, 1),
    ({"precision": 1, "pair_variant": 3, "i_per_thread": 2}, 3), ({"precision": 1, "pair_variant": 1}, 1)])
def test_the_kernel_used_is_reported(pn, kw, variant):
    x, v, m = _system(5000, 1)
    with pn.Context(5000, **{"eps": EPS, "inv_c2": 1e-2, **kw}) as c:
        c.set_state(x, v, m)
        c.force()
        assert c.stats().pair_variant == variant
