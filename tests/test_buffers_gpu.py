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
