"""The session's one context is in its default launch mode (plain launches, no graph
replay) whatever the tests before this file did with it: a chain takes as many
launches as on a context of its own.  A replayed chain takes one more, which sets
the step counter."""
import numpy as np
import pytest

from ed_solver_b200 import edk
from ed_solver_b200.model import matsubara, workload

pytestmark = pytest.mark.gpu


def _launches(c):
    import torch
    w = workload("c1")
    h = edk.Hamiltonian(c, w.model, 3, 3)
    x = torch.tensor(np.random.default_rng(0).normal(size=h.dim), device="cuda")
    run = lambda: h.green_chain(x, 12, -3.0, 1, matsubara(w.beta, 4))
    run()
    n = c.launches
    run()
    return c.launches - n


def test_shared_context_runs_plain_launches(ctx):
    own = edk.Context(0)
    try:
        plain = _launches(own)
        own.set_graphs(True)
        assert _launches(own) > plain
    finally:
        own.close()
    assert _launches(ctx) == plain
