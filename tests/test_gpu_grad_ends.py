"""Ends of the adjoint's recurrences: a right-hand side that vanishes (a sector of
one state), and more frequencies than the continued fraction's buffers hold at a
time."""
import numpy as np
import pytest

from ed_solver_b200 import edk
from ed_solver_b200.model import matsubara, star_model

pytestmark = pytest.mark.gpu


def _unit(n, i):
    import torch
    x = torch.zeros(n, dtype=torch.float64, device="cuda")
    x[i] = 1.0
    return x


def _occupied(m, h):
    from ed_solver_b200.edk import basis
    up = (basis(m.ns, h.nup).astype(np.int64) >> m.nb) & 1
    return np.tile(up, h.ddn)


def test_one_state_has_no_residual(ctx):
    """The empty sector: psibar is a multiple of psi, so the projected right-hand side is
    exactly zero, no iteration runs and the residual is 0, not 0/0."""
    m = star_model(-1.0, 2.0, [-0.5, 0.4], [0.4, 0.3])
    h = edk.Hamiltonian(ctx, m, 0, 0)
    wn = matsubara(10.0, 4)
    gbar = np.ones((1, 4), complex)
    grad, G, st = h.grad_green(_unit(1, 0), 0.0, [(0, 0, True)], 5, wn, gbar, edk.star_params(m))
    assert st["cg_iterations"] == 0 and st["cg_residual"] == 0.0
    assert np.isfinite(grad).all() and np.isfinite(G).all()


def test_many_frequencies_need_no_more_memory(ctx):
    """6e5 frequencies of a 100-step chain with 1 GB left on the device; only the first
    16 carry weight, so the gradient is that of those alone."""
    import torch
    m = star_model(-1.0, 2.0, np.linspace(-0.9, 0.8, 4), 0.2 + 0.05 * np.arange(4))
    h = edk.Hamiltonian(ctx, m, 2, 2)
    E, V = h.full_ed()
    psi = torch.tensor(V[:, 0].copy(), device="cuda")
    nw, params = 600_000, edk.star_params(m)
    wn, gbar = matsubara(10.0, nw), np.zeros((1, nw), complex)
    gbar[0, :16] = np.arange(16) - 3.0j
    few = h.grad_green(psi, float(E[0]), [(0, 0, True)], 100, wn[:16], gbar[:, :16], params, cg_tol=1e-12)
    torch.cuda.empty_cache()
    ctx.trim()
    hog = torch.empty(torch.cuda.mem_get_info()[0] - (1 << 30), dtype=torch.uint8, device="cuda")
    try:
        many = h.grad_green(psi, float(E[0]), [(0, 0, True)], 100, wn, gbar, params, cg_tol=1e-12)
    finally:
        del hog
        torch.cuda.empty_cache()
    assert np.array_equal(many[1][:, :16], few[1])
    assert np.abs(many[0] - few[0]).max() <= 1e-12 * np.abs(few[0]).max()
    z = 1j * wn[-1]                                  # the tail: G = <phi|phi> / z to order 1 / |z|
    assert abs(many[1][0, -1] * z - (V[:, 0] ** 2 @ (1 - _occupied(m, h)))) <= 20.0 / abs(z)
