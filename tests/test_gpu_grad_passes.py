"""The adjoint's device passes at their edges: <a|dH/dtheta|b> with fewer, as
many and more parameters than a block has warps, on rows of 1 to 126 columns,
against the oracle's operators (1e-12 relative); chains cut by the sector's
dimension (Krylov space exhausted) and of one step, and one to three frequencies,
against central differences of the oracle's own solve (1e-6 of the largest
component, h = 1e-5, as the bound of the long chains)."""
import numpy as np
import pytest
import torch

import oracle as O
from ed_solver_b200 import edk
from ed_solver_b200.model import AIMModel, matsubara, star_model

pytestmark = pytest.mark.gpu


def _one(m, p):
    z = AIMModel(m.nc, m.nb, np.zeros_like(m.ec), np.zeros_like(m.eb), np.zeros_like(m.vbc), np.zeros_like(m.u),
                 np.zeros_like(m.jj), 0.0, m.cutoff)
    return edk.perturb(z, p, 1.0)


@pytest.mark.parametrize("npar", [1, 3, 8, 9, 16, 17, 33])
@pytest.mark.parametrize("sec", [(0, 4), (1, 8), (4, 5)])
def test_bilinear_parameter_counts(ctx, npar, sec):
    rng = np.random.default_rng(npar)
    m = star_model(-1.0, 3.0, rng.uniform(-1, 1, 8), rng.uniform(0.2, 0.6, 8))
    params = (edk.star_params(m) + edk.star_params(m, 0) + edk.star_params(m, 1))[:npar]
    h = edk.Hamiltonian(ctx, m, *sec)
    a, b = rng.normal(size=(2, h.dim))
    got = h.dh_bilinear(torch.tensor(a, device="cuda"), torch.tensor(b, device="cuda"), params)
    for q, p in enumerate(params):
        ref = a @ O.OracleH(_one(m, p), *sec).hmult(b)
        assert abs(got[q] - ref) <= 1e-12 * max(1.0, np.linalg.norm(a) * np.linalg.norm(b)), (q, p)


def _loss(m, sec, chains, nit, wn, gbar, e0bar):
    E, V = np.linalg.eigh(O.OracleH(m, *sec).dense())
    val = e0bar * E[0]
    for c, (site, spin, dag) in enumerate(chains):
        phi, ts = O.apply_c(m, *sec, site, spin, dag, V[:, 0])
        G, _, _ = O.green_chain(O.OracleH(m, *ts), phi, nit, float(E[0]), 1 if dag else 2, wn, cutoff_dynamic=0.0)
        val += float(np.sum((np.conj(gbar[c]) * G).real))
    return val


@pytest.mark.parametrize("ns,sec,nit,nw", [(3, (1, 1), 50, 1), (4, (2, 2), 1, 3), (4, (2, 2), 2, 2), (5, (2, 3), 7, 33)])
def test_chain_lengths(ctx, ns, sec, nit, nw):
    rng = np.random.default_rng(ns)
    m = star_model(-0.8, 2.0, rng.uniform(-1, 1, ns - 1), rng.uniform(0.3, 0.6, ns - 1))
    params, chains, wn = edk.star_params(m), [(0, 0, True), (0, 1, False)], matsubara(20.0, nw)
    gbar = rng.normal(size=(2, nw)) + 1j * rng.normal(size=(2, nw))
    h = edk.Hamiltonian(ctx, m, *sec)
    E, V = h.full_ed()      # Lanczos stops at dim - 1 steps, short of the state in a 9-state sector
    grad, _, _ = h.grad_green(torch.tensor(V[:, 0].copy(), device="cuda"), float(E[0]), chains, nit, wn, gbar, params,
                              e0bar=0.4, cg_tol=1e-13)
    ref = np.array([(_loss(edk.perturb(m, p, 1e-5), sec, chains, nit, wn, gbar, 0.4) -
                     _loss(edk.perturb(m, p, -1e-5), sec, chains, nit, wn, gbar, 0.4)) / 2e-5 for p in params])
    assert np.abs(grad - ref).max() <= 1e-6 * np.abs(ref).max(), (grad, ref)
