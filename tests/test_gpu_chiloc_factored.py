"""The factored kernel of chi~_loc (matrix products over the cycle of the four
c+ elements) against the per-element kernel on the same inputs: sectors of
unequal sizes on both sides of the shared-memory limit, odd and single-state
sectors, degenerate energies and triples that take the vanishing-denominator
branches, and triples on the real axis, which keep the element-by-element
kernels.  Tolerance: |d| <= 1e-9 max|chi| of the batch, the bound the
reference is held to (FP64, another summation order)."""
import numpy as np
import pytest

from ed_solver_b200 import edk

pytestmark = pytest.mark.gpu

# (target, source) sectors of the fourteen matrices, in the order of chi_tilde_loc_'s arguments
PAIRS = [(1, 0), (2, 0), (7, 1), (7, 2), (5, 2), (0, 3), (8, 3), (0, 4), (9, 4), (2, 8), (1, 9), (4, 10), (3, 10), (4, 6)]


def _inputs(rng, dims, degenerate):
    E = [np.sort(np.round(rng.uniform(-2, 2, d), 1) if degenerate else rng.uniform(-2, 2, d)) for d in dims]
    M = [rng.standard_normal((dims[t], dims[s])) * (rng.random((dims[t], dims[s])) < 0.7) for t, s in PAIRS]
    return E, M


def _triples(beta):
    nu = lambda n: 1j * (2 * n + 1) * np.pi / beta
    return np.array([(nu(0), nu(1), nu(2)), (nu(0), nu(1), -nu(1)), (nu(2), -nu(2), nu(0)), (nu(-3), nu(1), nu(0)),
                     (nu(1), nu(-1), -nu(-1))])


def _both(ctx, E, M, w, ops=(1, 2)):
    out = []
    for plain in (False, True):
        edk.chiloc_set_kernel(plain)
        try:
            out.append(edk.chiloc(ctx, E, M, w, 10.0, 3.0, -2.0, 5, 2, 2, ops=ops))
        finally:
            edk.chiloc_set_kernel(False)
    return out


@pytest.mark.parametrize("degenerate", [False, True])
@pytest.mark.parametrize("dims", [[1] * 11, [2, 1, 3, 2, 1, 4, 1, 5, 2, 3, 1], [36, 24, 24, 24, 24, 6, 6, 16, 16, 16, 16],
                                  [37, 5, 33, 12, 31, 7, 4, 9, 36, 2, 17], [41, 20, 64, 1, 38, 30, 11, 50, 3, 27, 45]])
def test_factored_equals_per_element(ctx, dims, degenerate):
    rng = np.random.default_rng(sum(dims))
    E, M = _inputs(rng, dims, degenerate)
    new, old = _both(ctx, E, M, _triples(10.0))
    for a, b in zip(new, old):
        assert np.abs(a - b).max() <= 1e-9 * np.abs(b).max()
    only, _ = _both(ctx, E, M, _triples(10.0), ops=(2,))
    assert only[0] is None and np.array_equal(only[1], new[1])


def test_real_frequencies_keep_their_kernel(ctx):
    rng = np.random.default_rng(3)
    E, M = _inputs(rng, [6, 4, 4, 4, 4, 1, 1, 6, 6, 6, 6], False)
    w = np.array([(0.3, 0.7, -0.45), (0.9, -0.2 + 0.1j, 1.1)])
    new, old = _both(ctx, E, M, w)
    for a, b in zip(new, old):
        assert np.isfinite(b).all() and np.abs(a - b).max() <= 1e-9 * np.abs(b).max()
