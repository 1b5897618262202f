"""The first H*v of a sector issued inside a stream capture: no launch shape has
been timed yet and none can be, so the call takes one untimed, and timing waits for
a later call.  Sectors with and without Hund terms, both element types, against the
generic kernel, bit for bit in FP64."""
import numpy as np
import pytest

from ed_solver_b200 import edk
from ed_solver_b200.model import star_model

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["float64", "float32"])
@pytest.mark.parametrize("ns,nup,ndn,nc", [(11, 5, 5, 2), (8, 4, 4, 2), (11, 5, 5, 1)])
def test_first_product_inside_a_capture(ns, nup, ndn, nc, dtype):
    import torch
    rng = np.random.default_rng(ns + nc)
    nb = ns - nc
    m = star_model([-1.2, -0.8][:nc], 2.5, rng.uniform(-1.5, 1.5, nb), rng.uniform(0.2, 0.5, nb),
                   orbital_of_bath=[k % nc for k in range(nb)], nc=nc, Uprime=1.3, J=0.4 if nc == 2 else 0.0,
                   cutoff=1e-8)
    s = torch.cuda.Stream()
    ctx = edk.Context(0, stream=s)
    try:
        h = edk.Hamiltonian(ctx, m, nup, ndn)
        x = torch.tensor(rng.normal(size=h.dim), device="cuda", dtype=getattr(torch, dtype))
        y = torch.zeros_like(x)
        torch.cuda.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=s):
            h.hmult(x, out=y)
        g.replay()
        torch.cuda.synchronize()
        ctx.set_kernel_path(1)
        z = h.hmult(x)
        torch.cuda.synchronize()
        ctx.set_kernel_path(0)
        assert torch.equal(y, z) if dtype == "float64" else (y - z).abs().max() <= 2.0 ** -23 * z.abs().max()
        assert ctx.launches > 0 and h.launch_shape_chosen("f64" if dtype == "float64" else "f32", False) is None
        h.hmult(x, out=y)
        torch.cuda.synchronize()
        assert torch.equal(y, z) if dtype == "float64" else (y - z).abs().max() <= 2.0 ** -23 * z.abs().max()
        del g
    finally:
        ctx.close()
