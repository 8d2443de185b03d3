"""The autotuner on the GPU: every launch-shape candidate evaluates the same
expressions in the same order, so a tuned solve must be bit-identical to the
untuned one (and, in FP64, to the oracle); the table survives a save/load
round trip and an empty table restores the defaults."""
import ctypes as C

import numpy as np
import pytest

from code_only_b200 import abi, workloads as w
from code_only_b200.solver import FMGPoisson, SFMError
from tests.oracle_lib import oracle_solve
from tests.test_gpu_planes import box, face_nested

pytestmark = pytest.mark.gpu

CASES = {
    "amr3_periodic": (lambda: w.small_periodic(2, 8, 3, 1), w.gaussian_peak, abi.SFM_BC_PERIODIC, {}),
    "amr3_sphere_l4": (lambda: w.small_sphere(2, 8, 3, 2), w.softened_sphere, abi.SFM_BC_SPHERE,
                       {"zero_mean": 0, "lmax": 4}),
    "amr3_periodic_ni16": (lambda: w.small_periodic(2, 16, 3, 4), w.gaussian_peak, abi.SFM_BC_PERIODIC, {}),
}


@pytest.mark.parametrize("prec", [abi.SFM_PREC_FP64, abi.SFM_PREC_MIXED], ids=["fp64", "mixed"])
@pytest.mark.parametrize("name", list(CASES))
def test_tuned_solve_is_bitwise_unchanged(name, prec):
    mk, fn, bc, kw = CASES[name]
    h = mk()
    p = abi.default_params(bc, rel_tol=1e-10, max_outer=40, precision=prec, **kw)
    rho = w.block_field(h, p.ngh_io, fn)
    with FMGPoisson(h, params=p) as s:
        psi0, g0, st0 = s.solve(rho)
        s.autotune(2)
        table = s.tune_table()
        assert any(ln.startswith(("ghost_fill", "relax_threads", "resid_bpc")) for ln in table.splitlines())
        psi1, g1, st1 = s.solve(rho)
        s.load_tune_table("")
        assert s.tune_table().strip().splitlines()[1:] == []
        s.load_tune_table(table)
        assert s.tune_table() == table
        psi2, g2, st2 = s.solve(rho)
        with pytest.raises(SFMError):
            s.load_tune_table("relax_threads 4 8 -1 -1 100\n")
        assert s.tune_table() == table            # a rejected table leaves the old one
    assert np.array_equal(psi0, psi1) and np.array_equal(g0, g1)
    assert np.array_equal(psi0, psi2) and np.array_equal(g0, g2)
    assert st0.outer_iters == st1.outer_iters
    if prec == abi.SFM_PREC_FP64:
        _, psi_o, g_o, _, _ = oracle_solve(h, rho, abi.default_params(bc, rel_tol=1e-10, max_outer=40, **kw))
        assert np.array_equal(psi1[:, 1:-1, 1:-1, 1:-1], psi_o[:, 1:-1, 1:-1, 1:-1])


@pytest.mark.parametrize("name", list(CASES))
def test_tuned_mixed_schedule_keeps_the_fp64_solution(name):
    """With a density, sfm_autotune also tunes the schedule of the mixed
    path's FP32 inner solve (V-cycles, sweeps, base-grid corrections).  The
    FP64 defect correction still converges to the same potential: within
    1e-9 (max norm, relative; phi's mean removed on periodic boxes) of the
    FP64 oracle in phi and g, at relative residual <= 1e-10."""
    import torch
    mk, fn, bc, kw = CASES[name]
    h = mk()
    p = abi.default_params(bc, rel_tol=1e-10, max_outer=40, precision=abi.SFM_PREC_MIXED, **kw)
    rho = w.block_field(h, p.ngh_io, fn)
    rho_d = torch.from_numpy(rho).cuda()
    with FMGPoisson(h, params=p) as s:
        s.autotune(2, rho_d.data_ptr())
        table = s.tune_table()
        for knob in ("fmg_ncycle", "fmg_sweeps", "vmg_sweeps", "base_corrections", "fused_sweeps", "local_sweeps"):
            assert any(ln.startswith(knob + " 4 ") for ln in table.splitlines()), knob
        psi2, g2, st2 = s.solve(rho)
    assert st2.converged and st2.true_rel_residual <= 1e-10
    _, psi1, g1, _, _ = oracle_solve(h, rho, abi.default_params(bc, rel_tol=1e-10, max_outer=40, **kw))
    n = h.ni
    a, b = psi2[:, 2:2 + n, 2:2 + n, 2:2 + n], psi1[:, 2:2 + n, 2:2 + n, 2:2 + n]
    if bc == abi.SFM_BC_PERIODIC:
        a, b = a - a.mean(), b - b.mean()
    assert np.abs(a - b).max() / np.abs(b).max() <= 1e-9
    ga, gb = g2[:, :, 2:2 + n, 2:2 + n, 2:2 + n], g1[:, :, 2:2 + n, 2:2 + n, 2:2 + n]
    assert np.abs(ga - gb).max() / np.abs(gb).max() <= 1e-9


# with planes, and with ghost passes (k_relax_bulk)
FUSED_CASES = CASES | {
    "amr3_zmirror": (lambda: w.mirror_sphere(3, 8, 3), w.wide_sphere, abi.SFM_BC_ZMIRROR, {"zero_mean": 0}),
    "amr2_zmirror_ni16": (lambda: w.mirror_sphere(2, 16, 2), w.wide_sphere, abi.SFM_BC_ZMIRROR, {"zero_mean": 0}),
    "face_nested": (lambda: face_nested(8), w.gaussian_peak, abi.SFM_BC_PERIODIC, {}),
}


@pytest.mark.parametrize("mask,local", [(1, 1), (2, 1), (3, 1), (1, 2), (3, 2), (3, 3)])
@pytest.mark.parametrize("name", list(FUSED_CASES))
def test_fused_sweep_keeps_the_fp64_solution(name, mask, local):
    """fused_sweeps bit 0 makes every smoothing sweep of the mixed path's
    FP32 fmg_lin one launch for both colours (the second colour with the
    ghost cells and reflux fluxes of before the sweep), bit 1 the same for
    the sweeps of vmg_fas; local_sweeps 2 runs two full sweeps on the staged
    block per launch.  The FP64 defect correction must still reach the
    FP64 oracle's potential within 1e-9 at relative residual <= 1e-10, the
    profiled launches must report two colours each, and a solve after the
    table is cleared runs the two-launch sweep again (one colour each)."""
    mk, fn, bc, kw = FUSED_CASES[name]
    h = mk()
    p = abi.default_params(bc, rel_tol=1e-10, max_outer=40, precision=abi.SFM_PREC_MIXED, profile=1, **kw)
    rho = w.block_field(h, p.ngh_io, fn)
    with FMGPoisson(h, params=p) as s:
        s.load_tune_table(f"fused_sweeps 4 {h.ni} -1 -1 {mask}\nlocal_sweeps 4 {h.ni} -1 -1 {local}\n")
        psi2, g2, st2 = s.solve(rho)
        psi3, g3, _ = s.solve(rho)                     # the graph replayed
        s.load_tune_table("")
        _, _, st4 = s.solve(rho)
    assert st2.converged and st2.true_rel_residual <= 1e-10
    assert st2.smoother_colours == (2 * local if mask & 1 else 1) and st2.smoother_launches > 0
    assert st4.smoother_colours == 1
    assert np.array_equal(psi2, psi3) and np.array_equal(g2, g3)
    _, psi1, g1, _, _ = oracle_solve(h, rho, abi.default_params(bc, rel_tol=1e-10, max_outer=40, **kw))
    n = h.ni
    a, b = psi2[:, 2:2 + n, 2:2 + n, 2:2 + n], psi1[:, 2:2 + n, 2:2 + n, 2:2 + n]
    if bc == abi.SFM_BC_PERIODIC:
        a, b = a - a.mean(), b - b.mean()
    assert np.abs(a - b).max() / np.abs(b).max() <= 1e-9
    ga, gb = g2[:, :, 2:2 + n, 2:2 + n, 2:2 + n], g1[:, :, 2:2 + n, 2:2 + n, 2:2 + n]
    assert np.abs(ga - gb).max() / np.abs(gb).max() <= 1e-9


@pytest.mark.parametrize("nt", [256, 288, 512, 544])
@pytest.mark.parametrize("name", ["amr3_periodic", "amr3_periodic_ni16"])
def test_smoother_cta_sizes_are_bitwise(name, nt):
    """Every CTA size of the bulk-copy smoother (warp 0 producing, 7, 8, 15
    or 16 consumer warps) computes each cell with the same expression: the
    FP64 solve stays bit-identical to the oracle, and the mixed solve with
    fused sweeps is bit-identical to the one with the default CTA size."""
    mk, fn, bc, kw = CASES[name]
    h = mk()
    edges = [e for e in (4, 8, 16) if e <= h.ni]
    p64 = abi.default_params(bc, rel_tol=1e-10, max_outer=40, **kw)
    rho = w.block_field(h, p64.ngh_io, fn)
    with FMGPoisson(h, params=p64) as s:
        s.load_tune_table("".join(f"relax_threads 8 {e} -1 -1 {nt}\n" for e in edges))
        psi, _, _ = s.solve(rho)
    _, psi_o, _, _, _ = oracle_solve(h, rho, p64)
    assert np.array_equal(psi[:, 1:-1, 1:-1, 1:-1], psi_o[:, 1:-1, 1:-1, 1:-1])
    pmx = abi.default_params(bc, rel_tol=1e-10, max_outer=40, precision=abi.SFM_PREC_MIXED, **kw)
    fused = f"fused_sweeps 4 {h.ni} -1 -1 3\n"
    with FMGPoisson(h, params=pmx) as s:
        s.load_tune_table(fused)
        psi_a, g_a, _ = s.solve(rho)
        s.load_tune_table(fused + "".join(f"relax_threads 4 {e} -1 {k} {nt}\n" for e in edges for k in (-1, 1)))
        psi_b, g_b, _ = s.solve(rho)
    assert np.array_equal(psi_a, psi_b) and np.array_equal(g_a, g_b)


# boxes whose sweeps exchange planes, and those that keep the ghost passes
SMOOTHER_CASES = {
    "planes": (lambda: w.small_periodic(2, 8, 3, 1), w.gaussian_peak, abi.SFM_BC_PERIODIC, 32),
    "passes_zmirror": (lambda: w.mirror_sphere(3, 8, 3), w.wide_sphere, abi.SFM_BC_ZMIRROR, 0),
    "passes_face_nested": (lambda: face_nested(8), w.gaussian_peak, abi.SFM_BC_PERIODIC, 0),
    "passes_zmirror_ni16": (lambda: w.mirror_sphere(2, 16, 2), w.wide_sphere, abi.SFM_BC_ZMIRROR, 0),
}


@pytest.mark.parametrize("prec", [abi.SFM_PREC_FP64, abi.SFM_PREC_MIXED], ids=["fp64", "mixed"])
@pytest.mark.parametrize("name", list(SMOOTHER_CASES))
def test_smoother_launches_the_tables_cta_size(name, prec):
    """relax_threads sets the CTA size of whichever smoother serves a level,
    with planes or with ghost passes, and never a result bit."""
    mk, fn, bc, extra = SMOOTHER_CASES[name]
    h = mk()
    p = abi.default_params(bc, rel_tol=1e-10, max_outer=40, precision=prec, zero_mean=int(bc == abi.SFM_BC_PERIODIC))
    rho = w.block_field(h, p.ngh_io, fn)
    elem, kinds = (8, (-1,)) if prec == abi.SFM_PREC_FP64 else (4, (-1, 1))
    fused = "" if prec == abi.SFM_PREC_FP64 else f"fused_sweeps 4 {h.ni} -1 -1 3\n"
    with FMGPoisson(h, params=p) as s:
        lib = s.lib
        lib.sfm_debug_smoother_threads.argtypes = [C.c_void_p, C.c_int, C.c_int]

        def threads():
            return [lib.sfm_debug_smoother_threads(s.ctx, f, int(k > 0)) for f in range(h.ni.bit_length() - 2) for k in kinds]

        edges = [h.ni >> f for f in range(h.ni.bit_length() - 2)]   # down to 4
        assert threads() == [(512 if e >= 16 else 256) + extra for e in edges for _ in kinds]
        s.load_tune_table(fused)
        psi, g, _ = s.solve(rho)
        for nt in (256, 288, 512, 544):
            s.load_tune_table(fused + "".join(f"relax_threads {elem} {e} -1 {k} {nt}\n" for e in edges for k in kinds))
            assert threads() == [nt] * len(threads())
            psi2, g2, _ = s.solve(rho)
            assert np.array_equal(psi, psi2) and np.array_equal(g, g2)


def test_fused_sweep_is_ignored_in_fp64():
    """An FP64 context given fused_sweeps 1 still runs the reference's two
    colour launches and stays bit-identical to the oracle."""
    mk, fn, bc, kw = CASES["amr3_periodic"]
    h = mk()
    p = abi.default_params(bc, rel_tol=1e-10, max_outer=40, profile=1, **kw)
    rho = w.block_field(h, p.ngh_io, fn)
    with FMGPoisson(h, params=p) as s:
        s.load_tune_table(f"fused_sweeps 4 {h.ni} -1 -1 3\nfused_sweeps 8 {h.ni} -1 -1 3\n")
        psi2, _, st2 = s.solve(rho)
    assert st2.smoother_colours == 1
    _, psi1, _, _, _ = oracle_solve(h, rho, abi.default_params(bc, rel_tol=1e-10, max_outer=40, **kw))
    assert np.array_equal(psi2[:, 1:-1, 1:-1, 1:-1], psi1[:, 1:-1, 1:-1, 1:-1])


def test_fp64_context_keeps_the_reference_schedule():
    """The schedule knobs exist only for the mixed path: tuning an FP64
    context with a density adds none, and its solve stays bit-identical to
    the oracle."""
    import torch
    mk, fn, bc, kw = CASES["amr3_periodic"]
    h = mk()
    p = abi.default_params(bc, rel_tol=1e-10, max_outer=40, **kw)
    rho = w.block_field(h, p.ngh_io, fn)
    rho_d = torch.from_numpy(rho).cuda()
    with FMGPoisson(h, params=p) as s:
        s.autotune(2, rho_d.data_ptr())
        assert not any(ln.startswith(("fmg_ncycle", "fmg_sweeps", "vmg_sweeps", "base_corrections", "fused_sweeps",
                                      "local_sweeps"))
                       for ln in s.tune_table().splitlines())
        psi2, _, _ = s.solve(rho)
    _, psi1, _, _, _ = oracle_solve(h, rho, p)
    assert np.array_equal(psi2[:, 1:-1, 1:-1, 1:-1], psi1[:, 1:-1, 1:-1, 1:-1])


@pytest.fixture(scope="module")
def base64():
    """64^3 base grids (32^3 blocks of 4^3 cells), which k_mg_cycle serves"""
    out = {}
    for bc, fn in ((abi.SFM_BC_PERIODIC, w.gaussian_peak), (abi.SFM_BC_SPHERE, w.softened_sphere)):
        h = box(32, 4, bc)
        p = abi.default_params(bc, rel_tol=1e-10, max_outer=2, zero_mean=int(bc == abi.SFM_BC_PERIODIC))
        rho = w.block_field(h, p.ngh_io, fn)
        out[bc] = h, p, rho, oracle_solve(h, rho, p)
    return out


@pytest.mark.parametrize("nct,wide", [(1, 16), (2, 16), (4, 16), (8, 16), (8, 32), (16, 16), (16, 32), (4, 32), (4, 64),
                                      (16, 64)])
@pytest.mark.parametrize("bc", [abi.SFM_BC_PERIODIC, abi.SFM_BC_SPHERE], ids=["periodic", "isolated"])
def test_base_grid_cluster_is_bitwise(base64, bc, nct, wide):
    """k_mg_cycle as a cluster of CTAs (the large levels spread over every
    CTA, the small ones on CTA 0, the maxima over the cluster) computes every
    cell with the same expression: the FP64 solve stays bit-identical to the
    oracle whatever the shape.  A shape the GPU cannot hold resident falls
    back to one CTA, which must match as well."""
    h, p, rho, (_, psi_o, g_o, st_o, _) = base64[bc]
    with FMGPoisson(h, params=p) as s:
        s.load_tune_table(f"base_ctas 8 64 -1 -1 {nct}\nbase_wide 8 64 -1 -1 {wide}\n")
        psi, g, st = s.solve(rho)
        psi2, g2, _ = s.solve(rho)                       # the graph replayed
    assert st.outer_iters == st_o.outer_iters
    assert np.array_equal(psi[:, 1:-1, 1:-1, 1:-1], psi_o[:, 1:-1, 1:-1, 1:-1])
    n = h.ni
    assert np.array_equal(g[:, :, 2:2 + n, 2:2 + n, 2:2 + n], g_o[:, :, 2:2 + n, 2:2 + n, 2:2 + n])
    assert np.array_equal(psi, psi2) and np.array_equal(g, g2)


# base grids that k_mgs_cycle serves, and a shape of k_mg_cycle for each
SMALL_BASE_CASES = {
    "uniform128": (lambda: w.uniform_periodic(16, 8), 32, 16, 16),
    "amr_base16": (lambda: w.small_periodic(16, 8, 2, 3), 32, 4, 32),
    "uniform64": (lambda: w.uniform_periodic(8, 8), 16, 8, 16),
}


@pytest.mark.parametrize("name", list(SMALL_BASE_CASES))
def test_base_grid_rows_of_an_old_table_are_accepted(name):
    """Up to 32^3 cells the base grid has one launch shape: rows for it in a
    saved table load, and the FP64 solve is the oracle's."""
    mk, nbase, nct, wide = SMALL_BASE_CASES[name]
    h = mk()
    p = abi.default_params(abi.SFM_BC_PERIODIC, rel_tol=1e-10, max_outer=30)
    rho = w.block_field(h, p.ngh_io, w.gaussian_peak)
    _, psi_o, g_o, st_o, _ = oracle_solve(h, rho, p)
    table = f"base_ctas 8 {nbase} -1 -1 {nct}\nbase_wide 8 {nbase} -1 -1 {wide}\n"
    with FMGPoisson(h, params=p) as s:
        s.load_tune_table(table)
        assert sorted(s.tune_table().splitlines()[1:]) == sorted(table.splitlines())
        psi, g, st = s.solve(rho)
        psi2, g2, _ = s.solve(rho)                       # the graph replayed
    assert st.outer_iters == st_o.outer_iters
    assert np.array_equal(psi[:, 1:-1, 1:-1, 1:-1], psi_o[:, 1:-1, 1:-1, 1:-1])
    n = h.ni
    assert np.array_equal(g[:, :, 2:2 + n, 2:2 + n, 2:2 + n], g_o[:, :, 2:2 + n, 2:2 + n, 2:2 + n])
    assert np.array_equal(psi, psi2) and np.array_equal(g, g2)


@pytest.mark.parametrize("prec", [abi.SFM_PREC_FP64, abi.SFM_PREC_MIXED], ids=["fp64", "mixed"])
def test_autotuned_base_grid_choice_is_recorded(prec):
    """On a base grid of 64^3 cells, which k_mg_cycle serves, the tuner times
    its shapes and records one."""
    h = box(32, 4, abi.SFM_BC_PERIODIC)
    p = abi.default_params(abi.SFM_BC_PERIODIC, rel_tol=1e-10, max_outer=2, precision=prec)
    elem = 8 if prec == abi.SFM_PREC_FP64 else 4
    with FMGPoisson(h, params=p) as s:
        s.autotune(1)
        lines = s.tune_table().splitlines()
    assert any(ln.startswith(f"base_ctas {elem} 64 ") for ln in lines)
    assert any(ln.startswith(f"base_wide {elem} 64 ") for ln in lines)


@pytest.mark.parametrize("report", [0, 1])
@pytest.mark.parametrize("prec", [abi.SFM_PREC_FP64, abi.SFM_PREC_MIXED], ids=["fp64", "mixed"])
@pytest.mark.parametrize("name,planes,outer", [("planes", True, True), ("isolated", True, False),
                                               ("passes_zmirror", False, False)])
def test_tuner_times_what_the_solve_launches(name, planes, outer, prec, report):
    """Rows of kernels that a context's solves do not launch are absent: the
    tiled residual where planes serve (but for the reported residual), and
    the shapes of k_mg_cycle on a base grid that k_mgs_cycle serves."""
    mk, fn, bc, _ = (SMOOTHER_CASES | {"isolated": (lambda: w.small_sphere(2, 8, 3, 2), w.softened_sphere,
                                                    abi.SFM_BC_SPHERE, 0)})[name]
    h = mk()
    p = abi.default_params(bc, precision=prec, zero_mean=int(bc == abi.SFM_BC_PERIODIC), report_residual=report)
    with FMGPoisson(h, params=p) as s:
        s.autotune(1)
        rows = {tuple(ln.split()[:3]) for ln in s.tune_table().splitlines()[1:]}
    elem = "8" if prec == abi.SFM_PREC_FP64 else "4"
    want = set() if planes else {elem}       # the descent of fmg_lin
    if not outer or report:                  # the outer residual, the reported one
        want.add("8")
    assert {r[1] for r in rows if r[0] == "resid_bpc"} == want
    assert not any(r[0] in ("base_ctas", "base_wide") for r in rows)
    assert ("relax_threads", elem, "8") in rows
