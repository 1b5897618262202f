"""chi~_loc where the device has room for the element-by-element kernel's buffers
but not for the factored kernel's: the call gives the factored kernel's scratch back
before it falls back, and its result is that of a call with room."""
import numpy as np
import pytest

from ed_solver_b200 import edk

pytestmark = pytest.mark.gpu

NF = 4_000_000


def test_falls_back_without_the_scratch():
    import torch
    ctx = edk.Context(0)
    try:
        # op 1 of a one-site (0, 0) sector: two terms over the sectors i and pdn, one state each
        E = [np.array([0.3])] + [None] * 10
        E[2] = np.array([0.7])
        M = [None] * 14
        M[1] = np.array([[1.3]])
        beta = 10.0
        nu = 1j * (2 * (np.arange(NF) % 97) + 1) * np.pi / beta
        w = np.stack([nu, -nu, nu[::-1]], axis=1)
        call = lambda t: edk.chiloc(ctx, E, M, t, beta, 2.0, 0.0, 1, 0, 0, ops=(1,))[0]
        ref = call(w[:5000])
        torch.cuda.empty_cache()
        ctx.trim()
        # scratch of the factored kernel: 80 + 32 bytes a triple; without it 96
        free = torch.cuda.mem_get_info()[0]
        hog = torch.empty(free - 104 * NF, dtype=torch.uint8, device="cuda")
        left = torch.cuda.mem_get_info()[0]
        assert 97 * NF < left < 111 * NF
        got = call(w)
        assert np.abs(got[:5000] - ref).max() <= 1e-9 * np.abs(ref).max()
        assert torch.cuda.mem_get_info()[0] >= left - (8 << 20)
        del hog
    finally:
        ctx.close()
        torch.cuda.empty_cache()
