"""The lifetime and the size of a context's and an ensemble's work buffers."""
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


@pytest.mark.parametrize("precision,n", [(0, 2050), (1, 3001), (1, 9001), (1, 30001)])
def test_captured_force_outlives_other_calls(pn, precision, n):
    """A force evaluation that a caller captured on its own stream still finds its buffers after the energies
    and steps of the same context."""
    torch = pytest.importorskip("torch")
    x, v, m = _system(n)
    with pn.Context(n, eps=EPS, inv_c2=1e-6, precision=precision, dt=1e-3) as c:
        c.set_state(x, v, m)
        dx, dv, dm = (torch.tensor(q, device="cuda") for q in (x, v, m))
        da = torch.zeros(n, 3, dtype=torch.float64, device="cuda")
        s = torch.cuda.Stream()

        def run():
            c.force_device(n, dx.data_ptr(), dv.data_ptr(), dm.data_ptr(), da.data_ptr(), s.cuda_stream)

        with torch.cuda.stream(s):
            run()
            s.synchronize()
            a = da.clone()
            g = torch.cuda.CUDAGraph()
            with torch.cuda.graph(g, stream=s):
                run()
        free = torch.cuda.mem_get_info()[0]
        c.energy()
        c.steps_energy(2)
        c.steps(1)
        c.force()
        c.sync()
        assert torch.cuda.mem_get_info()[0] > free - (8 << 20)  # no sums beside the captured ones (graphs are small)
        da.zero_()
        torch.cuda.synchronize()
        g.replay()
        torch.cuda.synchronize()
        assert torch.equal(a, da)


@pytest.mark.parametrize("precision", [0, 1])
def test_a_context_allocates_what_it_uses(pn, precision):
    """State 152 bytes per particle, results and staging 80, BH-relative positions 24, packs 168, tile origins 2,
    partial sums 1; the fixed-point pack (208) only once its sweep runs."""
    torch = pytest.importorskip("torch")
    n = 1 << 20
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    with pn.Context(n, eps=EPS, precision=precision):
        taken = free - torch.cuda.mem_get_info()[0]
    assert taken <= 440 * n + (32 << 20)  # (allocations are rounded up to 2 MiB)


class _NoMemory:
    """Takes the GPU's free memory, but for a few MiB."""

    def __enter__(self):
        import torch
        self.held, size = [], torch.cuda.mem_get_info()[0]
        while size >= 2 << 20:
            try:
                self.held.append(torch.empty(size, dtype=torch.uint8, device="cuda"))
            except torch.cuda.OutOfMemoryError:
                size //= 2
            size = min(size, torch.cuda.mem_get_info()[0])
        return self

    def __exit__(self, *a):
        import torch
        self.held.clear()
        torch.cuda.empty_cache()


def test_no_memory_for_the_fixed_point_pack(pn):
    """The FP64 sweep takes over, and gives way again once there is memory and the parameters are set anew."""
    pytest.importorskip("torch")
    n = 40001
    x, v, m = _system(n)
    with pn.Context(n, eps=EPS, inv_c2=1e-2) as c:  # (its kernels are loaded)
        c.set_state(x, v, m)
        a = c.force()
        assert c.stats().pair_variant == 6
    with pn.Context(n, eps=EPS, inv_c2=1e-2, i_per_thread=1, grid_split=16) as c:  # (so are its sums)
        c.set_state(x, v, m)
        b = c.force()
        with _NoMemory():
            c.set_params(i_per_thread=0, grid_split=0)
            d = c.force()
            assert c.stats().pair_variant == 1
        c.set_params()
        assert np.array_equal(c.force(), a) and c.stats().pair_variant == 6
    for f in (b, d):
        assert (np.linalg.norm(f - a, axis=1) <= 1e-12 * np.linalg.norm(a, axis=1).max()).all()


def test_no_memory_for_the_unordered_sweep(pn):
    """The packed sweep takes over, also while shapes are tuned (none is kept for the sweep that did not run), and
    gives way again once there is memory."""
    pytest.importorskip("torch")
    n = 20001
    x, v, m = _system(n)
    kw = dict(eps=EPS, inv_c2=1e-2, precision=1)
    with pn.Context(n, **kw) as c:
        c.set_state(x, v, m)
        a = c.force()
        assert c.stats().pair_variant == 5
    try:
        with pn.Context(n, grid_split=32, **kw) as c:  # (its sums are allocated)
            c.set_state(x, v, m)
            c.force()
            c.autotune(1)  # (every kernel is loaded)
            pn.lib().pn_autotune_clear()
        with pn.Context(n, grid_split=32, **kw) as c:
            c.set_state(x, v, m)
            c.force()
            with _NoMemory():
                c.set_params(grid_split=0)
                b = c.force()
                assert c.stats().pair_variant in (2, 3)
                c.autotune(1)
                c.force()
                assert c.stats().pair_variant != 5
            c.set_params(dt=1e-3)
            c.force()
            assert c.stats().pair_variant != 5  # (a tuned shape)
            pn.lib().pn_autotune_clear()
            c.set_params(dt=2e-3)
            assert np.array_equal(c.force(), a) and c.stats().pair_variant == 5
    finally:
        pn.lib().pn_autotune_clear()
    assert np.sqrt(((a - b) ** 2).sum() / (a ** 2).sum()) <= 2e-6  # (each within 1e-6 of FP64)


class _Cluster:
    def __init__(self, n):
        self.x, self.v, self.m = _system(n)


def test_ensemble_gives_its_sums_back(pn):
    """The partial sums of the unordered sweep (150 MB here) go when another sweep is asked for."""
    torch = pytest.importorskip("torch")
    clusters = [_Cluster(16385) for _ in range(4)]
    with pn.Ensemble(clusters, [EPS] * 4, precision=1, inv_c2=1e-2, dt=1e-3) as e:
        e.steps(1)
        e.get_state()
        free = torch.cuda.mem_get_info()[0]
        e.set_shape(2, 1)
        assert torch.cuda.mem_get_info()[0] - free > 100 << 20
        e.steps(1)
        e.get_state()


REFUSED = r"""
import sys
import numpy as np
import torch
import pn_gb300 as pn
sys.path.insert(0, sys.argv[1])
from test_buffers_gpu import EPS, _system
for precision, kw, variant in ((0, dict(i_per_thread=1, grid_split=32), 6), (1, dict(grid_split=32), 5)):
    n = 9001
    x, v, m = _system(n)
    with pn.Context(n, eps=EPS, inv_c2=1e-2, precision=precision, **kw) as c:
        c.set_state(x, v, m)
        c.force()
        c.set_params(**{k: 0 for k in kw})
        d = [torch.tensor(q, device="cuda") for q in (x, v, m)]
        a = torch.zeros(n, 3, dtype=torch.float64, device="cuda")
        s = torch.cuda.Stream()
        refused = None
        try:
            with torch.cuda.graph(torch.cuda.CUDAGraph(), stream=s):  # (capture that allows no allocation)
                try:
                    c.force_device(n, *(q.data_ptr() for q in d), a.data_ptr(), s.cuda_stream)
                except pn.PNError as e:
                    refused = e.status
        except RuntimeError:
            pass
        assert refused == -2, refused
        c.force()
        assert c.stats().pair_variant == variant
print("ok")
"""


def test_an_allocation_refused_while_capturing_is_an_error(pn):
    """... and no reason to take a slower sweep from then on.  (In a process of its own: the capture is broken off.)"""
    pytest.importorskip("torch")
    import os
    import subprocess
    import sys
    here = os.path.dirname(os.path.abspath(__file__))
    env = dict(os.environ, PYTHONPATH=os.path.dirname(here))
    r = subprocess.run([sys.executable, "-c", REFUSED, here], env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stderr
