"""The row kernels with Hund terms at the edges of their dispatch: sectors on
both sides of the size where shapes are timed, even and odd rows, table widths 8,
12 and 16, every launch shape, against the generic row kernel, bit for bit in
FP64 (one rounding of the output in FP32); unaligned vectors; a short chain's
coefficients; rows whose elements are infinite."""
import numpy as np
import pytest

from ed_solver_b200 import edk
from ed_solver_b200.model import matsubara, star_model

pytestmark = pytest.mark.gpu


def _model(ns):
    rng = np.random.default_rng(ns)
    nb = ns - 2
    m = star_model([-1.2, -0.8], 2.5, rng.uniform(-1.5, 1.5, nb), rng.uniform(0.2, 0.5, nb),
                   orbital_of_bath=[k % 2 for k in range(nb)], nc=2, Uprime=1.3, J=0.4, cutoff=1e-8)
    m.ec[:, 0, 1] = m.ec[:, 1, 0] = 0.15
    return m


@pytest.mark.parametrize("ns,nup,ndn", [(3, 1, 2), (5, 2, 2), (6, 0, 3), (7, 7, 3), (8, 4, 4), (11, 5, 5), (11, 6, 5),
                                        (12, 4, 6), (14, 4, 3), (15, 2, 13), (15, 3, 3)])
def test_hund_shapes_agree(ctx, ns, nup, ndn):
    import torch
    h = edk.Hamiltonian(ctx, _model(ns), nup, ndn)
    rng = np.random.default_rng(ns + nup)
    x = torch.tensor(rng.normal(size=h.dim), device="cuda")
    buf = torch.zeros(2 * h.dim + 2, dtype=torch.float64, device="cuda")
    odd, out = buf[1:h.dim + 1], torch.zeros(h.dim + 1, dtype=torch.float64, device="cuda")[1:]
    odd.copy_(x)
    big = x.clone()
    big[:: max(1, h.dim // 7)] = np.inf
    wn = matsubara(20.0, 8)
    try:
        ctx.set_kernel_path(1)
        y, yf, yb = h.hmult(x), h.hmult(x.float()), h.hmult(big)
        al = h.green_chain(x, 6, -1.0, 1, wn)[1] if h.dim > 6 else None
        n = len(h.launch_shapes("f64")), len(h.launch_shapes("f32"))
        assert min(n) >= 1
        for path in [0] + [16 + i for i in range(max(n))]:
            ctx.set_kernel_path(path)
            assert torch.equal(h.hmult(x), y)
            if path < 16 + n[0]:
                assert torch.equal(torch.nan_to_num(h.hmult(big)), torch.nan_to_num(yb))
            assert (h.hmult(x.float()) - yf).abs().max() <= 2.0 ** -23 * y.abs().max()
            if al is not None:
                assert np.abs(h.green_chain(x, 6, -1.0, 1, wn)[1] - al).max() <= 1e-12 * np.abs(al).max()
        ctx.set_kernel_path(0)
        assert torch.equal(h.hmult(odd, out=out), y)
    finally:
        ctx.set_kernel_path(0)
