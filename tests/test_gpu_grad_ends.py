"""Ends of the adjoint's recurrences: a right-hand side that vanishes (a sector of
one state), a chain that breaks down long before its last step, and more
frequencies than the continued fraction's buffers hold at a time."""
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


def test_chain_stops_soon_after_a_breakdown(ctx):
    """No hybridisation: c+|basis state> is an eigenstate and the chain ends after one
    step.  The launches of a call do not grow with the steps it was allowed."""
    m = star_model(-1.0, 2.0, np.linspace(-0.9, 0.8, 9), np.zeros(9))
    h = edk.Hamiltonian(ctx, m, 5, 5)
    wn, params = matsubara(10.0, 8), edk.star_params(m)
    psi, gbar = _unit(h.dim, 0), np.ones((1, 8), complex)     # the impurity is the highest orbital: empty in state 0
    e0, out = float(h.hmult(psi)[0]), []
    for steps in (4, 4, 800):
        n0 = ctx.launches
        grad, G, st = h.grad_green(psi, e0, [(0, 0, True)], steps, wn, gbar, params)
        out.append((grad, G, st["forward_steps"], ctx.launches - n0))
    assert [o[2] for o in out] == [1, 1, 1]
    assert np.array_equal(out[1][0], out[2][0]) and np.array_equal(out[1][1], out[2][1])
    assert out[2][3] <= out[1][3] + 4 * 3 * 45                # at most three segments of sqrt(2 * 800) + 1 steps


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
