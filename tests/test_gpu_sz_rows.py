"""The Nambu row kernels at the edges of their dispatch: rows on both sides of
256 and 400 columns, few and many particles (rows far below the longest and near
it), one and two impurity orbitals, both term orders, against the kernel that
walks the whole term list, bit for bit in FP64; FP32 vectors within one rounding
of the output; unaligned vectors; a short chain's coefficients."""
import numpy as np
import pytest

from ed_solver_b200 import edk
from ed_solver_b200.model import NambuModel, matsubara, nambu_workload, star_model

pytestmark = pytest.mark.gpu


def _model(ns, nc, on_fly):
    if nc == 1:
        return nambu_workload(ns, seed=ns, on_fly=on_fly)
    rng = np.random.default_rng(ns)
    nb = ns - nc
    base = star_model([-1.2, -0.8], 2.5, rng.uniform(-1.5, 1.5, nb), rng.uniform(0.2, 0.5, nb),
                      orbital_of_bath=[k % 2 for k in range(nb)], nc=2, Uprime=1.3, J=0.0, cutoff=1e-8)
    base.ec[:, 0, 1] = base.ec[:, 1, 0] = 0.15
    pv = np.zeros((2, nb, 2))
    pv[0, 0, 0], pv[1, 2, 1] = 0.11, -0.09
    return NambuModel(base, np.diag(rng.uniform(0.1, 0.3, nb)), pv, on_fly)


@pytest.mark.parametrize("on_fly", [False, True])
@pytest.mark.parametrize("ns,npart,nc", [(4, 0, 1), (4, 8, 1), (6, 5, 2), (9, 9, 1), (10, 11, 1), (11, 1, 1), (11, 5, 1),
                                         (11, 11, 2), (12, 12, 1), (12, 23, 1), (13, 4, 1), (13, 14, 1)])
def test_row_kernels_agree(ctx, ns, npart, nc, on_fly):
    import torch
    h = edk.HamiltonianSz(ctx, _model(ns, nc, on_fly), npart)
    rng = np.random.default_rng(npart)
    x = torch.tensor(rng.normal(size=h.dim), device="cuda")
    buf = torch.zeros(2 * h.dim + 2, dtype=torch.float64, device="cuda")
    odd, out = buf[1:h.dim + 1], torch.zeros(h.dim + 1, dtype=torch.float64, device="cuda")[1:]
    odd.copy_(x)
    wn = matsubara(20.0, 8)
    try:
        ctx.set_kernel_path(1)
        y, yf = h.hmult(x), h.hmult(x.float())
        al = h.green_chain(x, 6, -1.0, 1, wn)[1] if h.dim > 6 else None
        ctx.set_kernel_path(0)
        assert torch.equal(h.hmult(x), y)
        assert torch.equal(h.hmult(odd, out=out), y)
        assert (h.hmult(x.float()) - yf).abs().max() <= 2.0 ** -23 * y.abs().max()
        if al is not None:
            assert np.abs(h.green_chain(x, 6, -1.0, 1, wn)[1] - al).max() <= 1e-12 * np.abs(al).max()
    finally:
        ctx.set_kernel_path(0)
