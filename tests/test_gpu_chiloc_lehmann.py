"""chi~_loc of the three kernels against the oracle's Lehmann sum, which shares no list
of terms with them: random sector data at every boundary case of (nup, ndn), with
degenerate energies and triples that take the vanishing-denominator branches.  A triple
on the real axis in the batch keeps a call on the split kernel.  Tolerance: 1000
roundings of the magnitudes added up (the sums are some hundred terms deep)."""
import numpy as np
import pytest

import oracle as O
from ed_solver_b200 import edk

pytestmark = pytest.mark.gpu

SITES = 3


def _inputs(rng, nup, ndn, degenerate):
    from math import comb
    E, M = [None] * 11, [None] * 14
    for q, (du, dd) in enumerate(O.CHILOC_SECTORS):
        nu, nd = nup + du, ndn + dd
        if 0 <= nu <= SITES and 0 <= nd <= SITES:
            e = rng.uniform(-2, 2, comb(SITES, nu) * comb(SITES, nd))
            E[q] = np.sort(np.round(e, 1) if degenerate else e)
    for q, (t, s, _) in enumerate(O.CHILOC_MATRICES):
        if E[t] is not None and E[s] is not None:
            M[q] = rng.standard_normal((len(E[t]), len(E[s]))) * (rng.random((len(E[t]), len(E[s]))) < 0.7)
    return E, M


@pytest.mark.parametrize("degenerate", [False, True])
@pytest.mark.parametrize("nup,ndn", [(1, 1), (0, 0), (3, 3), (0, 3), (3, 0), (1, 2), (2, 1), (2, 2)])
@pytest.mark.parametrize("kernel", ["factored", "split", "per-element"])
def test_kernels_against_the_lehmann_sum(ctx, kernel, nup, ndn, degenerate):
    E, M = _inputs(np.random.default_rng(10 * nup + ndn), nup, ndn, degenerate)
    beta, Z, gs, eps = 7.0, 3.0, min(e.min() for e in E if e is not None), 1e-5
    nu = lambda n: 1j * (2 * n + 1) * np.pi / beta
    w = [(nu(0), nu(1), nu(2)), (nu(0), nu(1), -nu(1)), (nu(2), -nu(2), nu(0)), (nu(1), nu(-1), -nu(-1))]
    ref = [[O.chiloc_lehmann(op, t, eps, beta, Z, gs, E, M) for t in w] for op in (1, 2)]
    edk.chiloc_set_kernel(kernel == "per-element")
    try:
        out = edk.chiloc(ctx, E, M, w + [(0.37, 1.3, -0.9)] * (kernel == "split"), beta, Z, gs, SITES, nup, ndn,
                         phi_eps=eps)
    finally:
        edk.chiloc_set_kernel(False)
    for got, want in zip(out, ref):
        for g, (v, scale) in zip(got, want):
            assert abs(g - v) <= 1e3 * 2.0**-53 * scale
