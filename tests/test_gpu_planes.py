"""The plane exchange of the sweeps, the V-cycle by lanes and the base-grid
multigrid in shared memory at the edges of their ranges: block edges 4, 8 and
16 with block counts that leave tiles partly filled, base grids of 2^3 to
64^3 cells under each boundary, base levels that are not a power of two (and
above the size one CTA averages), and a hierarchy nested over faces only,
whose margins the plane exchange does not serve.  FP64 must equal the oracle
bit for bit (the same expressions in the same order); mixed precision ends
within 1e-9 of it (both stop at a relative residual of 1e-10)."""
import ctypes as C

import numpy as np
import pytest

from code_only_b200 import abi, workloads as w
from code_only_b200.solver import FMGPoisson
from tests.oracle_lib import oracle_solve

pytestmark = pytest.mark.gpu

PER, SPH, ZM, CYL = abi.SFM_BC_PERIODIC, abi.SFM_BC_SPHERE, abi.SFM_BC_ZMIRROR, abi.SFM_BC_CYL_ZPERIODIC
DENSITY = {PER: w.gaussian_peak, SPH: w.softened_sphere, ZM: w.wide_sphere, CYL: w.beaded_line}


def box(nbase, ni, bc, corner=False):
    """nbase^3 blocks, one of them refined when corner is set"""
    periodic = {PER: True, SPH: False, ZM: False, CYL: (False, False, True)}[bc]
    lo = {PER: (0.0, 0.0, 0.0), ZM: (-0.5, -0.5, 0.0)}.get(bc, (-0.5, -0.5, -0.5))
    return w.build_hierarchy((nbase,) * 3, ni, 2 if corner else 1,
                             lambda L, q, g: (q == 0).all(axis=1) if corner else np.zeros(len(q), bool), periodic,
                             box_lo=lo, box_size=1.0)


def face_nested(ni):
    """One corner child of a refined base block refined again, nested over the
    six faces only: the coarse block next to it across a face has coarser
    neighbours, so that a margin is itself a coarse-fine ghost."""
    keep, w._NEIGH26 = w._NEIGH26, w._NEIGH26[np.abs(w._NEIGH26).sum(axis=1) == 1]
    try:
        h = w.build_hierarchy((6,) * 3, ni, 3, lambda L, q, g: (q == (2 if L == 0 else 5)).all(axis=1), True)
    finally:
        w._NEIGH26 = keep
    at = {tuple(q) for q in h.ijk[h.level == 1]}
    assert (6, 5, 5) in at and (6, 6, 5) not in at
    return h


CASES = {
    # block edges and partly filled tiles
    "ni4_amr3_base3": (lambda: w.small_periodic(3, 4, 3, 2), PER),
    "ni8_amr3_base5": (lambda: w.small_periodic(5, 8, 3, 5), PER),
    "ni16_amr2_base3_isolated": (lambda: w.small_sphere(3, 16, 2, 1), SPH),
    "ni8_amr4_base3_isolated": (lambda: w.small_sphere(3, 8, 4, 7), SPH),
    "ni8_corner_cylinder": (lambda: w.zperiodic_cylinder(4, 8, 3), CYL),
    "one_block_ni4": (lambda: box(1, 4, PER), PER),
    "one_block_ni16_isolated": (lambda: box(1, 16, SPH), SPH),
    # margins with another source: the ghost passes
    "face_nested_ni8": (lambda: face_nested(8), PER),
    # base grids of 2 n cells per edge, n base blocks of 2^3 cells there
    **{f"base_{bc}_{n}": (lambda n=n, bc=bc: box(n, 4, bc), bc) for n in (1, 2, 4, 8, 16) for bc in (PER, SPH, ZM, CYL)},
}


def run_both(h, bc, prec, **kw):
    p = abi.default_params(bc, precision=prec, zero_mean=1 if bc == PER else 0, **{**dict(rel_tol=1e-10, max_outer=40), **kw})
    rho = w.block_field(h, p.ngh_io, DENSITY[bc])
    with FMGPoisson(h, params=p) as s:
        psi, g, _ = s.solve(rho, allow_unconverged=True)
    po = abi.default_params(bc, zero_mean=p.zero_mean, rel_tol=p.rel_tol, max_outer=p.max_outer)
    _, psi_o, g_o, _, _ = oracle_solve(h, rho, po)
    n, gw = h.ni, p.ngh_io
    c = (Ellipsis,) + (slice(gw, gw + n),) * 3
    return psi[c], psi_o[c], g[c], g_o[c]


def check(h, bc, prec, **kw):
    psi, psi_o, g, g_o = run_both(h, bc, prec, **kw)
    if prec == abi.SFM_PREC_FP64:
        assert np.array_equal(psi, psi_o) and np.array_equal(g, g_o)
        return
    if bc == PER:   # the constant is free
        psi, psi_o = psi - psi.mean(), psi_o - psi_o.mean()
    assert np.abs(psi - psi_o).max() <= 1e-9 * np.abs(psi_o).max()
    assert np.abs(g - g_o).max() <= 1e-9 * np.abs(g_o).max()


@pytest.mark.parametrize("prec", [abi.SFM_PREC_FP64, abi.SFM_PREC_MIXED], ids=["fp64", "mixed"])
@pytest.mark.parametrize("name", list(CASES))
def test_edges_match_oracle(name, prec):
    mk, bc = CASES[name]
    check(mk(), bc, prec)


@pytest.mark.parametrize("nbase", [17, 32])
def test_large_base_levels_match_oracle(nbase):
    """17^3 base blocks: not a power of two and more than one CTA averages;
    32^3: a base grid of 64^3 cells, beyond the shared-memory cycle"""
    check(box(nbase, 4, PER), PER, abi.SFM_PREC_FP64, max_outer=2)


# hierarchy, and the device bytes that a context of it held in FP64 and in
# mixed precision when every sweep had ghost passes and every base grid
# k_mg_cycle
BYTES = {
    "ni4_amr3": (lambda: w.small_periodic(2, 4, 3, 1), PER, 3714264, 2691288),
    "ni8_amr3": (lambda: w.small_periodic(2, 8, 3, 1), PER, 16088280, 11609304),
    "ni16_amr3": (lambda: w.small_periodic(2, 16, 3, 4), PER, 89927248, 65292880),
    "ni32_amr2": (lambda: w.small_periodic(2, 32, 2, 0), PER, 87937936, 64164752),
    "ni8_amr3_isolated": (lambda: w.small_sphere(2, 8, 3, 2), SPH, 21651936, 15845856),
    "ni8_cylinder": (lambda: w.zperiodic_cylinder(2, 8, 3), CYL, 15748040, 11600840),
    "ni8_zmirror": (lambda: w.mirror_sphere(3, 8, 3), ZM, 12500816, 9784400),
    "uniform64": (lambda: w.uniform_periodic(8, 8), PER, 38202696, 27585864),
    "base5_ni4": (lambda: w.uniform_periodic(5, 4), PER, 2112616, 1520616),
    "one_block_ni4": (lambda: w.uniform_periodic(1, 4), PER, 21448, 16712),
    "one_block_ni16": (lambda: w.uniform_periodic(1, 16), PER, 422344, 308296),
}


@pytest.mark.parametrize("name", list(BYTES))
def test_planes_cost_no_device_memory(name):
    """The planes take the place of arrays that only the ghost passes or
    k_mg_cycle read: a context is no larger with them, so that what fitted a
    device before still does."""
    mk, bc, fp64, mixed = BYTES[name]
    h = mk()
    for prec, most in ((abi.SFM_PREC_FP64, fp64), (abi.SFM_PREC_MIXED, mixed)):
        with FMGPoisson(h, params=abi.default_params(bc, precision=prec, zero_mean=int(bc == PER))) as s:
            assert s.info()["device_bytes"] <= most


@pytest.mark.parametrize("stage", [4, 16 + 4], ids=["whole_arrays", "as_solved"])
def test_solve_after_stage_dump_is_unchanged(stage):
    """Stage dumps complete arrays a solve leaves unread; a solve on the same
    context before and after one gives the same bits."""
    h = w.small_periodic(3, 8, 3, 1)
    p = abi.default_params(PER, rel_tol=1e-10, max_outer=40)
    rho = w.block_field(h, p.ngh_io, w.gaussian_peak)
    lib = abi.load_library()
    lib.sfm_debug_solve.argtypes = [C.c_void_p, C.c_void_p, C.c_void_p, C.c_void_p, C.POINTER(abi.SfmStats),
                                    C.c_int, C.c_void_p]
    with FMGPoisson(h, params=p) as s:
        psi, g, _ = s.solve(rho)
        dump, start = np.zeros((h.nblocks,) + (h.ni + 2,) * 3), np.zeros_like(rho)
        assert lib.sfm_debug_solve(s.ctx, rho.ctypes.data, start.ctypes.data, None, None, stage,
                                   dump.ctypes.data) == 0
        psi2, g2, _ = s.solve(rho)
    assert np.array_equal(psi, psi2) and np.array_equal(g, g2)


@pytest.mark.parametrize("n", [2, 4, 8, 16, 32])
def test_noalloc_sizes_match_fourier_solution(n):
    """Every size of the allocation-free solve against the 7-point problem's
    exact solution: a residual of 1e-12 max|source| leaves an error below
    1e-12 |source| / lambda_min = 1e-12 x 100 x phi (lambda_min = 4 pi^2 and
    the source's norm at most 4 sin^2 n^2 x 3 = 12 n^2 times phi's: n = 32
    gives 3e-10)."""
    import torch
    rng = np.random.default_rng(n)
    rho = 1.0 + rng.random((n, n, n))
    k2 = (2.0 * n * np.sin(np.pi * np.arange(n) / n)) ** 2
    lam = -(k2[:, None, None] + k2[None, :, None] + k2[None, None, :])
    lam[0, 0, 0] = 1.0
    src = np.fft.fftn(4.0 * np.pi * (rho - rho.mean())) / lam
    src[0, 0, 0] = 0.0
    phi = np.fft.ifftn(src).real
    f = abi.load_library().sfm_uniform_solve_noalloc
    f.argtypes = [C.c_void_p, C.c_void_p, C.c_int, C.c_double, C.c_double, C.c_double, C.c_int, C.POINTER(C.c_int),
                  C.POINTER(C.c_double), C.c_void_p]
    f.restype = C.c_int
    rho_d = torch.from_numpy(rho).cuda()
    psi = torch.full_like(rho_d, float("nan"))
    cycles, rr = C.c_int(), C.c_double()
    assert f(rho_d.data_ptr(), psi.data_ptr(), n, 1.0 / n, 4.0 * np.pi, 1e-12, 200, C.byref(cycles), C.byref(rr),
             torch.cuda.current_stream().cuda_stream) == abi.SFM_OK
    out = psi.cpu().numpy()
    assert np.abs(out - out.mean() - phi).max() <= 1e-9 * np.abs(phi).max()
