"""Plain H*v and the fused steps have a launch shape each, timed on the first call of
either, kept for the handle and for others of the sector's shape; inside a capture
H*v takes the steps' shape untimed.  Results are those of the generic row kernel, bit
for bit."""
import numpy as np
import pytest

from ed_solver_b200 import edk
from ed_solver_b200.model import matsubara, star_model

pytestmark = pytest.mark.gpu


def _model(ns, nc):
    rng = np.random.default_rng(ns)
    nb = ns - nc
    return star_model([-1.2, -0.8][:nc], 2.5, rng.uniform(-1.5, 1.5, nb), rng.uniform(0.2, 0.5, nb),
                      orbital_of_bath=[k % nc for k in range(nb)], nc=nc, Uprime=1.3, J=0.4 if nc == 2 else 0.0)


@pytest.mark.parametrize("ns,nc,sec", [(8, 1, (4, 4)), (11, 1, (5, 5)), (11, 2, (5, 5))])
@pytest.mark.parametrize("first", ["step", "hv"])
def test_each_mode_is_timed_once(first, ns, nc, sec):
    import torch
    c = edk.Context(0)
    try:
        hs = [edk.Hamiltonian(c, _model(ns, nc), *sec) for _ in range(2)]
        x = torch.tensor(np.random.default_rng(1).normal(size=hs[0].dim), device="cuda")
        c.set_kernel_path(1)
        ref = hs[0].hmult(x).clone()
        c.set_kernel_path(0)
        calls = {"step": lambda h: h.green_chain(x, 5, -3.0, 1, matsubara(20.0, 4)), "hv": lambda h: h.hmult(x)}

        def launches(mode, h):
            n = c.launches
            calls[mode](h)
            return c.launches - n

        assert len(hs[0].launch_shapes("f64")) > 1
        for mode in (first, "hv" if first == "step" else "step"):
            cold = launches(mode, hs[0])
            warm = launches(mode, hs[0])
            assert cold > warm and launches(mode, hs[1]) == warm
        assert torch.equal(hs[0].hmult(x), ref) and torch.equal(hs[1].hmult(x), ref)
        assert launches("hv", hs[0]) == 1
    finally:
        c.close()


@pytest.mark.parametrize("ns,sec", [(8, (4, 4)), (11, (6, 5))])
def test_first_chain_ends_at_once(ns, sec):
    """The shapes are timed on a vector whose Krylov space is itself: no step of the timing
    may take the chain for ended."""
    import torch
    m = star_model([-1.2], 2.5, np.linspace(-1.5, 1.5, ns - 1), np.zeros(ns - 1))
    wn, out = matsubara(20.0, 8), []
    for path in (0, 1):
        c = edk.Context(0)
        try:
            h = edk.Hamiltonian(c, m, *sec)
            c.set_kernel_path(path)
            x = torch.zeros(h.dim, dtype=torch.float64, device="cuda")
            x[h.dim // 3] = 1.0
            out.append(h.green_chain(x, 5, -3.0, 1, wn)[0])
            e = float(h.hmult(x)[h.dim // 3])
        finally:
            c.close()
        assert np.abs(out[-1] - 1.0 / (1j * wn - (e + 3.0))).max() <= 1e-12
    assert np.array_equal(out[0], out[1])


@pytest.mark.parametrize("same", [True, False])
def test_capture_after_steps_is_not_timed(same):
    import torch
    s = torch.cuda.Stream()
    c = edk.Context(0, stream=s)
    try:
        h = [edk.Hamiltonian(c, _model(11, 1), 5, 5) for _ in range(2)]
        x = torch.tensor(np.random.default_rng(1).normal(size=h[0].dim), device="cuda")
        y = torch.zeros_like(x)
        torch.cuda.synchronize()
        h[0].green_chain(x, 5, -3.0, 1, matsubara(20.0, 4))
        torch.cuda.synchronize()
        g, n = torch.cuda.CUDAGraph(), c.launches
        with torch.cuda.graph(g, stream=s):
            h[0 if same else 1].hmult(x, out=y)
        assert c.launches - n == 1
        g.replay()
        c.set_kernel_path(1)
        ref = h[0].hmult(x)
        torch.cuda.synchronize()
        assert torch.equal(y, ref)
        del g
    finally:
        c.close()
