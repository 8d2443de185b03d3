"""What a call leaves on which stream: work that another stream or another
call could overtake."""
import numpy as np
import pytest

from code_only_b200 import abi, workloads as w
from code_only_b200.solver import FMGPoisson

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [abi.SFM_PREC_FP64, abi.SFM_PREC_MIXED], ids=["fp64", "mixed"])
def test_create_leaves_nothing_on_the_default_stream(prec):
    """A context's tables and its plane of zeros are in place when sfm_create
    returns, whatever the legacy default stream is doing: behind a kernel that
    keeps that stream busy, a create returns while the kernel still runs, and
    the solve that follows equals one on an idle GPU.  (Set-up work queued on
    the default stream would hold the create back, or end after it returned
    and be overtaken by the solve, whose stream does not wait for that one.)"""
    import torch
    h = w.small_sphere(2, 8, 3, 2)
    p = abi.default_params(abi.SFM_BC_SPHERE, rel_tol=1e-10, max_outer=40, zero_mean=0, precision=prec)
    rho = w.block_field(h, p.ngh_io, w.softened_sphere)
    with FMGPoisson(h, params=p) as s:   # loads every kernel
        psi, g, _ = s.solve(rho)
    torch.cuda.synchronize()
    done = torch.cuda.Event()
    default = torch.cuda.default_stream()
    with torch.cuda.stream(default):
        torch.cuda._sleep(int(2e9))   # about a second
        done.record(default)
    with FMGPoisson(h, params=p) as s:
        held_back = done.query()
        psi2, g2, _ = s.solve(rho)
    assert not held_back
    assert np.array_equal(psi, psi2) and np.array_equal(g, g2)
