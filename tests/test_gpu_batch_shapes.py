"""Batched chains with every block size and every number of blocks per chain that is
feasible (the tuner's choice depends on timing), against the same chains one after the
other: fewer rows than blocks, rows up to the 32 KB that a block stages, rows beyond
them (6,435 elements: 51 KB in FP64), Hund terms.  Every chain runs all its steps."""
import numpy as np
import pytest

from ed_solver_b200 import edk
from ed_solver_b200.model import matsubara, star_model

pytestmark = pytest.mark.gpu

STEPS = 12


@pytest.mark.parametrize("dtype", ["f64", "f32"])
@pytest.mark.parametrize("ns,nc,sectors,copies", [(6, 2, [(3, 3), (5, 2)], 3), (8, 1, [(4, 3)], 40), (14, 1, [(7, 1)], 1),
                                                  (15, 1, [(7, 1), (8, 2)], 1)])
def test_every_batch_shape_equals_single_chains(ctx, ns, nc, sectors, copies, dtype):
    import torch
    rng = np.random.default_rng(ns)
    m = star_model([-1.2, -0.8][:nc], 2.5, rng.uniform(-1.5, 1.5, ns - nc), rng.uniform(0.2, 0.5, ns - nc),
                   orbital_of_bath=[k % nc for k in range(ns - nc)], nc=nc, Uprime=1.3, J=0.4 if nc == 2 else 0.0)
    wn, chains = matsubara(20.0, 8), []
    for sec in sectors:
        h = edk.Hamiltonian(ctx, m, *sec)
        for i in range(copies):
            x = torch.tensor(rng.normal(size=h.dim), device="cuda", dtype=getattr(torch, "float" + dtype[1:]))
            chains.append(dict(h=h, start=x, e0=-6.0, iph=1 + i % 2, weight=0.5 ** (i % 4), out=i % 2))
    G0, s0 = edk.green_batch(ctx, chains, STEPS, wn, 2, mode=1, dtype=dtype)
    assert s0["steps"] == STEPS * len(chains)
    tol, shapes = 1e-10 if dtype == "f64" else 2e-5, set()      # FP32: the vectors' roundings differ
    try:
        for i in range(15):
            ctx.set_kernel_path(16 + i)
            G, st = edk.green_batch(ctx, chains, STEPS, wn, 2, mode=0, dtype=dtype)
            shapes.add((st["block"], st["blocks_per_sm"]))
            assert st["steps"] == s0["steps"] and st["tuned_shapes"] == 0
            assert np.abs(G - G0).max() <= tol * np.abs(G0).max(), i
    finally:
        ctx.set_kernel_path(0)
    assert {b for b, _ in shapes} == {128, 256, 512}
