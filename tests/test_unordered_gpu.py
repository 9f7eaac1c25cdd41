"""The mixed sweep over unordered pairs: every star's sums, and which sweep an ensemble takes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = 0.02


class _Cluster:
    def __init__(self, n):
        rng = np.random.default_rng(n)
        self.x = rng.uniform(-1, 1, (n, 3))
        self.v = rng.normal(0, 0.3, (n, 3))
        self.m = rng.uniform(0.5, 1.5, n) / n
        self.m[0] = 0.02


def _magnitudes(s):
    """The sum of the magnitudes of a star's terms: its pairs' and the BH's."""
    import torch
    x, m = torch.tensor(s.x, device="cuda"), torch.tensor(s.m, device="cuda")
    out = torch.empty_like(m)
    for i in range(0, len(m), 2048):
        r2 = ((x[None] - x[i:i + 2048, None]) ** 2).sum(2)
        out[i:i + 2048] = (m * r2.sqrt() * (r2 + EPS * EPS) ** -1.5).sum(1)
    return out.cpu().numpy()


@pytest.mark.parametrize("n", [8001, 8129, 9001, 12289, 20001])
def test_every_star(pn, n):
    """Each star within 1e-6 of the sum of its terms' magnitudes (a term's FP32 roundings, below 16 u): faint stars
    and single rows too, among them stars of 1e-6 of the others' mass and of 1e3 times it."""
    pytest.importorskip("torch")
    s = _Cluster(n)
    s.m[5:n:97] *= 1e-6
    s.m[7:n:501] *= 1e3
    s.x[11:n:301] *= 30.0
    out = []
    for precision in (1, 0):
        with pn.Context(n, eps=EPS, inv_c2=1e-6, precision=precision) as c:
            c.set_state(s.x, s.v, s.m)
            out.append(c.force())
            assert c.stats().pair_variant == (5 if precision else 6)
    err = np.linalg.norm(out[0] - out[1], axis=1)
    assert (err[1:] <= 1e-6 * _magnitudes(s)[1:]).all()


@pytest.mark.parametrize("sizes,unordered", [
    ([16385] * 3, True),      # large clusters
    ([1001] * 4, True),       # few small ones: the packed sweep's items would leave SMs idle
    ([401] * 200, False),     # many small ones
    ([65537] * 4, False),     # partial sums beyond 2 GB
])
def test_the_sweep_of_an_ensemble(pn, sizes, unordered):
    """Which sweep ran shows in the last bits: the shape of the size class given as it was selects the packed one."""
    clusters = [_Cluster(sizes[0])] * len(sizes)
    k = (sizes[0] - 1).bit_length() - 1
    with pn.Ensemble(clusters, [EPS] * len(sizes), precision=1, inv_c2=1e-2, dt=1e-3) as e:
        a = e.force()
        _, _, tile_j, tiles = e.shape(k)
        e.set_shape(size_class=k, tile_j=tile_j, tiles_per_item=tiles)
        b = e.force()
    assert all(np.array_equal(p, q) for p, q in zip(a, b)) == (not unordered)
    for p, q in zip(a, b):
        assert np.sqrt(((p - q) ** 2).sum() / (q ** 2).sum()) <= 2e-6  # (each within 1e-6)
