"""Shapes of the mixed Newtonian and energy sweeps on either side of their rules' lines, against the FP64 path.

Tolerance 1e-6 of the RMS acceleration, as for the other mixed shapes; the energies against the same sweep in
a given shape (a star's pair with itself is rounded to FP32 in both)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = 0.02


def _system(n):
    rng = np.random.default_rng(n)
    x = rng.uniform(-1, 1, (n, 3))
    v = rng.normal(0, 0.3, (n, 3))
    m = rng.uniform(0.5, 1.5, n) / n
    m[0] = 0.02
    return x, v, m


def _run(pn, s, **kw):
    with pn.Context(len(s[0]), eps=EPS, inv_c2=0.0, **kw) as c:
        c.set_state(*s)
        a = c.force()
        st = c.stats()
        return a, np.array(c.energy()), (st.i_per_thread, st.tile_j, st.grid_split)


@pytest.mark.parametrize("nstar", [11999, 12000, 15999, 16000, 20000, 37000, 65535, 65536])
def test_light_sweeps(pn, nstar):
    s = _system(nstar + 1)
    a, e, shape = _run(pn, s, precision=1)
    if 16000 <= nstar < 65536:  # two stars per thread, four tiles per split, 32 splits at most
        assert shape == (2, 256, min(32, (nstar + 255) // 256 // 4, -(-8 * 4 * 152 // ((nstar + 255) // 256))))
    elif nstar >= 12000:
        assert shape[0] == 2
    b, _, _ = _run(pn, s)
    assert np.sqrt(((a - b) ** 2).sum() / (b ** 2).sum()) <= 1e-6
    _, f, _ = _run(pn, s, precision=1, pair_variant=2, i_per_thread=1, tile_j=64)
    assert np.abs(e - f).max() <= 1e-6 * np.abs(f).max()
