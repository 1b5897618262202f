"""Batched chains shared out over clusters of blocks: one chain and many, sectors
with fewer rows than a cluster has blocks and with rows longer than the staging
buffer, chains that end early, Hund terms, FP32 vectors, against the same chains
run one after the other."""
import numpy as np
import pytest

from ed_solver_b200 import edk
from ed_solver_b200.model import matsubara, star_model

pytestmark = pytest.mark.gpu


def _model(ns, nc):
    rng = np.random.default_rng(ns)
    nb = ns - nc
    return star_model([-1.2, -0.8][:nc], 2.5, rng.uniform(-1.5, 1.5, nb), rng.uniform(0.2, 0.5, nb),
                      orbital_of_bath=[k % nc for k in range(nb)], nc=nc, Uprime=1.3, J=0.4 if nc == 2 else 0.0,
                      cutoff=1e-8)


@pytest.mark.parametrize("dtype", ["f64", "f32"])
@pytest.mark.parametrize("ns,nc,sectors,copies", [(3, 1, [(1, 1), (0, 2), (3, 0)], 1), (5, 2, [(2, 2)], 1),
                                                  (6, 2, [(3, 3), (5, 1), (0, 3)], 5), (8, 2, [(4, 4)], 2),
                                                  (8, 1, [(4, 3), (1, 7)], 150), (14, 1, [(7, 1), (1, 6)], 1)])
def test_clusters_equal_single_chains(ctx, ns, nc, sectors, copies, dtype):
    import torch
    m, wn, chains = _model(ns, nc), matsubara(20.0, 16), []
    rng = np.random.default_rng(ns)
    for sec in sectors:
        h = edk.Hamiltonian(ctx, m, *sec)
        for i in range(copies):
            x = torch.tensor(rng.normal(size=h.dim), device="cuda", dtype=getattr(torch, "float" + dtype[1:]))
            chains.append(dict(h=h, start=x * (i != 3), e0=-6.0, iph=1 + i % 2, weight=0.5 ** (i % 4), out=i % 2))
    G0, s0 = edk.green_batch(ctx, chains, 25, wn, 2, mode=1, dtype=dtype)
    G, st = edk.green_batch(ctx, chains, 25, wn, 2, mode=0, dtype=dtype)
    tol = 1e-10 if dtype == "f64" else 2e-5       # FP32: the vectors' roundings differ
    assert np.abs(G - G0).max() <= tol * np.abs(G0).max()
    assert st["chains"] == s0["chains"] and st["steps"] <= s0["steps"] + 25 * len(chains)
