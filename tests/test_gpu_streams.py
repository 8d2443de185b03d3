"""What a call leaves on which stream: work that another stream or another
call could overtake."""
import ctypes as C

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


def test_noalloc_calls_without_outputs_leave_the_result_words_alone():
    """Calls that ask for no host outputs may overlap one that does: it still
    reports its own cycles, residual and status.  The queue of another stream
    is kept full of calls that stop at once (no cycles allowed, a residual of
    1) while asking calls run and copy their result words."""
    import torch
    f = abi.load_library().sfm_uniform_solve_noalloc
    f.argtypes = [C.c_void_p, C.c_void_p, C.c_int, C.c_double, C.c_double, C.c_double, C.c_int, C.POINTER(C.c_int),
                  C.POINTER(C.c_double), C.c_void_p]
    f.restype = C.c_int
    rng = np.random.default_rng(5)
    asks, other = torch.cuda.Stream(), torch.cuda.Stream()
    rho = [torch.from_numpy(rng.random((n, n, n))).cuda() for n in (4, 2)]
    psi = [torch.empty_like(r) for r in rho]
    torch.cuda.synchronize()

    def ask():
        cycles, rr = C.c_int(-7), C.c_double(-7.0)
        rc = f(rho[0].data_ptr(), psi[0].data_ptr(), 4, 0.25, 1.0, 1e-9, 100, C.byref(cycles), C.byref(rr),
               asks.cuda_stream)
        return rc, cycles.value, rr.value

    alone = ask()
    assert alone[0] == abi.SFM_OK and alone[1] > 0
    got, open_ = [], torch.cuda.Event()
    for _ in range(20):
        with torch.cuda.stream(other):
            torch.cuda._sleep(int(4e7))   # about 20 ms: holds the calls back until all are queued
            open_.record(other)
        for _ in range(500):
            assert f(rho[1].data_ptr(), psi[1].data_ptr(), 2, 0.5, 1.0, 1e-9, 0, None, None,
                     other.cuda_stream) == abi.SFM_OK
        open_.synchronize()
        got += [ask() for _ in range(20)]
    torch.cuda.synchronize()
    assert set(got) == {alone}
