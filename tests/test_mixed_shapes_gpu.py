"""The mixed force sweep over unordered pairs and the launch shapes that the library chooses by itself,
at the edges of their tiles, row blocks and panels, against the FP64 path.

Tolerance 1e-6 of the RMS acceleration (normwise): a pair term takes some 12 FP32 roundings on top of
its inverse distance (3 units), its sum up to 128 more in a tile, of random sign: less than 16 u = 1e-6."""
import os
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = 0.02

# The unordered sweep's shape for every size class comes from a table of tuned shapes, which a process
# reads once.
SMALL = r"""
import sys
import numpy as np
import pn_gb300 as pn
sys.path.insert(0, sys.argv[1])
from test_mixed_shapes_gpu import close, force, system
for n in (2, 3, 128, 129, 130, 512, 513, 514, 641, 1026, 2049, 4100):
    x, v, m = system(n)
    for ic2 in (1e-6, 1.0):
        with pn.Context(n + 300, eps=0.02, inv_c2=ic2, precision=1, dt=1e-3) as c:
            c.set_state(x, v, m)
            a = c.force()
            assert c.stats().pair_variant == 5
            assert np.array_equal(a, c.force())
            c.steps(1)
            x1, v1 = c.get_state()
            close(c.force(), force(pn, x1, v1, m, ic2, 0), n)
        close(a, force(pn, x, v, m, ic2, 0), n)
print("ok")
"""


def system(n):
    rng = np.random.default_rng(n)
    x = rng.uniform(-1, 1, (n, 3))
    v = rng.normal(0, 0.3, (n, 3))
    m = rng.uniform(0.5, 1.5, n) / n
    m[0] = 0.02
    return x, v, m


def force(pn, x, v, m, ic2, precision, **kw):
    with pn.Context(len(x), eps=EPS, inv_c2=ic2, precision=precision, **kw) as c:
        c.set_state(x, v, m)
        return c.force()


def close(a, b, what=None):
    e = np.sqrt(((a - b) ** 2).sum() / (b ** 2).sum())
    assert e <= 1e-6, (what, e)


@pytest.mark.parametrize("tiles", [1, 3])
def test_every_pair_once(tmp_path, tiles):
    table = tmp_path / "shapes"
    table.write_text("".join(f"1 1 {c} 4 1 128 {tiles} 4 1.0\n" for c in range(13)))
    here = os.path.dirname(os.path.abspath(__file__))
    env = dict(os.environ, PN_TUNE_CACHE=str(table), PYTHONPATH=os.path.dirname(here))
    r = subprocess.run([sys.executable, "-c", SMALL, here], env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stderr


@pytest.mark.parametrize("ic2", [0.0, 1e-6, 1.0])
@pytest.mark.parametrize("n", [2, 129, 130, 257, 1026, 4099, 8000, 8002, 9001, 70001])
def test_chosen_shapes(pn, n, ic2):
    x, v, m = system(n)
    with pn.Context(n, eps=EPS, inv_c2=ic2, precision=1, dt=1e-3) as c:
        c.set_state(x, v, m)
        a, st = c.force(), c.stats()
        assert (st.pair_variant == 5) == (n > 8000 and ic2 != 0)
        assert (st.grid_split > 1) or n < 70001 or ic2 == 0  # several panels
        e = np.array(c.energy())
    with pn.Context(n, eps=EPS, inv_c2=ic2) as c:
        c.set_state(x, v, m)
        close(a, c.force())
    # the energy against the same sweep in a given shape (a star's pair with itself, m / eps, is rounded
    # to FP32 like every term and taken off in FP64, in both)
    with pn.Context(n, eps=EPS, inv_c2=ic2, precision=1, pair_variant=2, i_per_thread=1, tile_j=64) as c:
        c.set_state(x, v, m)
        f = np.array(c.energy())
    assert np.abs(e - f).max() <= 1e-6 * np.abs(f).max()


def test_buffers_grow_between_steps(pn):
    """A captured step stays valid when later calls of other sizes and kinds need larger buffers."""
    x, v, m = system(9001)
    with pn.Context(20001, eps=EPS, inv_c2=1e-6, precision=1, dt=1e-3) as c:
        c.set_state(x, v, m)
        c.steps(2)
        c.energy()
        c.steps_energy(1)
        c.steps(1)
        got = c.get_state()
        c.set_state(*system(20001))
        c.steps(1)
        c.force()
        c.set_state(x, v, m)
        c.steps(4)
        again = c.get_state()
    assert np.abs(got[0] - again[0]).max() <= 1e-9 and np.abs(got[1] - again[1]).max() <= 1e-7


@pytest.mark.parametrize("precision", [0, 1])
def test_tuned_shapes(pn, precision):
    """A tuned context gives the results of the chosen shape."""
    x, v, m = system(5000)
    out = []
    try:
        for tune in (False, True):
            with pn.Context(5000, eps=EPS, inv_c2=1.0, precision=precision) as c:
                c.set_state(x, v, m)
                if tune:
                    c.autotune(3)
                out.append((c.force(), np.array(c.energy())))
    finally:
        pn.lib().pn_autotune_clear()
    (a, e), (b, f) = out
    if precision:
        close(b, a)
    else:
        assert np.abs(a - b).max() <= 1e-12 * np.abs(a).max()
    assert np.abs(e - f).max() <= (1e-6 if precision else 1e-12) * np.abs(e).max()


class _System:
    def __init__(self, n):
        self.x, self.v, self.m = system(n)


@pytest.mark.parametrize("ic2", [1e-6, 1.0])
def test_ensemble_every_pair_once(pn, ic2):
    """Clusters at the edges of tiles and row blocks in one launch, also after their energies and with the
    shape given (which selects the ordered sweep)."""
    sizes = [1, 2, 3, 128, 129, 130, 512, 513, 514, 641, 1026, 2049, 4100]
    systems = [_System(n) for n in sizes]
    with pn.Ensemble(systems, [EPS] * len(sizes), precision=1, inv_c2=ic2, dt=1e-3) as e:
        a = e.force()
        en = e.energy()
        again = e.force()
        e.set_shape(2, 1)
        ordered = e.force()
        en2 = e.energy()
    for s, f, g, h in zip(systems, a, again, ordered):
        assert np.array_equal(f, g)
        ref = force(pn, s.x, s.v, s.m, ic2, 0)
        if len(s.x) > 1:
            close(f, ref, len(s.x))
            close(h, ref, len(s.x))
    assert np.abs(en - en2).max() <= 1e-6 * np.abs(en).max()
