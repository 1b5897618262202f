"""A Nambu sector created on one stream and used on another: every table is in
place when the creation returns, whatever the first stream still has queued.
H*v on the second stream equals the kernel that walks the term list, which reads
none of the row kernels' tables, bit for bit (FP64)."""
import pytest

from ed_solver_b200 import edk
from ed_solver_b200.model import nambu_workload

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ns,npart", [(5, 5), (10, 11), (13, 13)])    # row kernel: short rows, staged; wide kernel
def test_sector_created_on_another_stream(ns, npart):
    import ctypes as C

    import torch
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    ctx = edk.Context(0, stream=a)
    try:
        m = nambu_workload(ns, seed=ns, on_fly=False)
        g = torch.Generator(device="cuda").manual_seed(ns)
        h = edk.HamiltonianSz(ctx, m, npart)
        edk.lib().edk_ctx_set_stream(ctx.h, C.c_void_p(b.cuda_stream))
        assert a.query()                                  # nothing of the creation is still queued
        x = torch.randn(h.dim, generator=g, device="cuda", dtype=torch.float64)
        torch.cuda.current_stream().synchronize()
        y = h.hmult(x)
        b.synchronize()
        ctx.set_kernel_path(1)
        z = h.hmult(x)
        b.synchronize()
        assert torch.equal(y, z)
    finally:
        ctx.close()
