"""The oracle's Lehmann sum for chi~_loc against Wick's theorem: without interaction
the sum over all sectors is beta G(w1) G(w3) (delta_{w1+w2} - delta_{w2+w3}) for equal
spins and beta G_up(w1) G_dn(w3) delta_{w1+w2} for different ones.  The matrices of c+_dn leave out the up electrons that it passes; the
theorem wants them.  Tolerance: 1000 roundings of the magnitudes added up (the sums are
some hundred terms deep)."""
import numpy as np
import pytest

import oracle as O
from ed_solver_b200.model import star_model


def _inputs(m, nup, ndn):
    E, M, _ = O.chiloc_inputs(m, nup, ndn)
    for q, (_, s, spin) in enumerate(O.CHILOC_MATRICES):
        if spin == 1 and M[q] is not None:
            M[q] = M[q] * (-1) ** (nup + O.CHILOC_SECTORS[s][0])
    return E, M


@pytest.mark.parametrize("op", [1, 2])
def test_noninteracting_sum_is_wicks(op):
    m, beta, eps = star_model(-0.3, 0.0, [-0.45, 0.7], [0.4, 0.5]), 6.0, 1e-5
    ns, nu = m.ns, lambda n: 1j * (2 * n + 1) * np.pi / beta
    sectors = [(a, b) for a in range(ns + 1) for b in range(ns + 1)]
    data = {s: _inputs(m, *s) for s in sectors}
    es = np.concatenate([data[s][0][0] for s in sectors])
    gs, Z = es.min(), np.exp(-beta * (es - es.min())).sum()
    green = lambda z, spin: O.lehmann_green(m, sectors, beta, np.array([z.imag]), spin=spin)[0]
    for w in [(nu(0), nu(1), nu(2)), (nu(1), -nu(1), nu(0)), (nu(0), nu(1), -nu(1)), (nu(2), -nu(2), nu(2))]:
        got, scale = 0j, 0.0
        for s in sectors:
            v, c = O.chiloc_lehmann(op, w, eps, beta, Z, gs, *data[s])
            got, scale = got + v, scale + c
        same = abs(w[0] + w[1]) < eps
        wick = beta * green(w[0], 1 if op == 1 else 0) * green(w[2], 1) * \
            (same - (abs(w[1] + w[2]) < eps if op == 1 else 0))
        assert abs(got - wick) <= 1e3 * 2.0**-53 * scale, (w, got, wick, scale)
