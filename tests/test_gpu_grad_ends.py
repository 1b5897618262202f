"""Ends of the adjoint's recurrences: a right-hand side that vanishes (a sector of
one state)."""
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
