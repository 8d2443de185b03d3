"""Performance cases of the self-gravity solver: what a host program has it do.

Each case is one call (or one time step's call) through the public entry
points: sfm_solve_device / sfm_solve / sfm_adjoint on a context that the
program keeps while its hierarchy is unchanged, the allocation-free uniform
solve, and the device-side linking after a regrid.  Hierarchies come from
code_only_b200.workloads; a density is the workload's own profile times a
seeded smooth modulation, so that every seed is another source on the same
blocks, as in a run whose hierarchy outlives a few steps.
"""
from __future__ import annotations

import ctypes
import functools
import math
import random

import numpy as np
import torch

from code_only_b200 import abi, workloads as w
from code_only_b200.solver import FMGPoisson, link_blocks

# The schedule and launch shapes sfm_autotune chooses for the Jeans-refined
# hierarchies of 8^3 blocks in mixed precision, kept as a program keeps the
# table of sfm_tune_save from its first run: fused colour sweeps, two per
# launch, one V-cycle of three sweeps, the base grid as a cluster.
TUNED = "\n".join([
    "fused_sweeps 4 8 -1 -1 3", "local_sweeps 4 8 -1 -1 2", "fmg_ncycle 4 8 -1 -1 1", "fmg_sweeps 4 8 -1 -1 3",
    "vmg_sweeps 4 8 -1 -1 2", "base_corrections 4 8 -1 -1 10", "relax_threads 4 8 -1 1 288",
    "relax_threads 4 4 -1 1 288", "resid_bpc 4 8 -1 -1 4", "resid_bpc 8 8 -1 -1 2",
    "base_ctas 4 32 -1 -1 16", "base_wide 4 32 -1 -1 16", "base_ctas 4 16 -1 -1 8", "base_wide 4 16 -1 -1 16", ""])


def listed():
    solve = dict(kind="solve", host=False, warm=False, tol=1e-10, table=False)
    return [
        # the smallest call: a code inside a fixed pool solves its uniform
        # 32^3 box without allocating anything
        dict(name="noalloc32", kind="noalloc", n=32, tol=1e-10),
        # plain FP64 on one uniform periodic level of 64^3 cells, the
        # reference's own gravity test size: launch latency decides
        dict(solve, name="uniform64_fp64", shape="uniform", nbase=8, ni=8, nlev=1, prec=abi.SFM_PREC_FP64),
        # a uniform 128^3 box in 16^3 blocks, mixed precision as it comes
        dict(solve, name="uniform128_b16_mixed", shape="uniform", nbase=8, ni=16, nlev=1, prec=abi.SFM_PREC_MIXED),
        # a collapse on concentric levels with the isolated boundary: few
        # blocks on many levels, in both precisions
        dict(solve, name="nested5_fp64", shape="nested", nbase=8, ni=8, nlev=5, prec=abi.SFM_PREC_FP64),
        dict(solve, name="nested5_mixed_tuned", shape="nested", nbase=8, ni=8, nlev=5, prec=abi.SFM_PREC_MIXED,
             table=True),
        # a base box that is not a power of two (no base-grid multigrid)
        dict(solve, name="nested3_base6_fp64", shape="nested", nbase=6, ni=8, nlev=3, prec=abi.SFM_PREC_FP64,
             tol=1e-6),
        # one time step of a host code as the reference calls it: host
        # arrays, the last step's potential as warm start, tolerance 1e-3
        dict(solve, name="step_host_fp64", shape="cloud", nbase=8, ni=8, nlev=3, prec=abi.SFM_PREC_FP64, host=True,
             warm=True, tol=1e-3),
        # the turbulent cloud refined to six levels by the Jeans rule (the
        # benchmark): 133,856 blocks, uneven level counts
        dict(solve, name="jeans6_fp64", shape="cloud", nbase=16, ni=8, nlev=6, prec=abi.SFM_PREC_FP64),
        dict(solve, name="jeans6_mixed_tuned", shape="cloud", nbase=16, ni=8, nlev=6, prec=abi.SFM_PREC_MIXED,
             table=True),
        # the same kind of cloud in 16^3 blocks, the layout of deep runs
        dict(solve, name="cloud3_b16_mixed", shape="cloud", nbase=8, ni=16, nlev=3, prec=abi.SFM_PREC_MIXED),
        # gradient of a functional of phi for an inverse problem
        dict(name="adjoint_nested4", kind="adjoint", shape="nested", nbase=8, ni=8, nlev=4,
             prec=abi.SFM_PREC_MIXED, tol=1e-8),
        # links of all blocks after a regrid, blocks in the order they come
        dict(name="link_jeans6", kind="link", shape="cloud", nbase=16, ni=8, nlev=6),
    ]


def draw(rng: random.Random):
    kind = rng.choice(["noalloc", "solve", "solve", "solve", "solve", "solve", "adjoint", "link"])
    if kind == "noalloc":
        return dict(kind="noalloc", n=rng.choice([2, 4, 8, 16, 32]), tol=10.0 ** -rng.randint(4, 11))
    if kind == "link":
        return dict(kind="link", shape="cloud", nbase=rng.choice([4, 5, 6, 7, 8, 12, 16]), ni=8, nlev=rng.randint(1, 5))
    shape = rng.choice(["uniform", "nested", "cloud", "sparse", "sparse_sphere"] + (["cylinder"] if kind == "solve" else []))
    if kind == "adjoint" and shape == "cloud":
        shape = "sparse"
    ni = rng.choice([4, 8, 8, 8, 16])
    if shape == "uniform":
        nbase, nlev = rng.choice([1, 2, 3, 4, 5, 6, 8, 16]), 1
    elif shape == "cloud":
        nbase, nlev = rng.choice([4, 8, 8]), rng.randint(2, 4)
        ni = 8 if nlev > 3 else ni
    elif shape in ("sparse", "sparse_sphere"):
        nbase, nlev = rng.choice([2, 3, 4, 5, 6]), rng.randint(2, 4)
    else:
        nbase, nlev = rng.choice([4, 6, 8]), rng.randint(2, 5)
    if ni == 16:
        nbase, nlev = min(nbase, 8), min(nlev, 3)
    prec = rng.choice([abi.SFM_PREC_FP64, abi.SFM_PREC_MIXED])
    if kind == "adjoint":
        return dict(kind=kind, shape=shape, nbase=min(nbase, 6), ni=min(ni, 8), nlev=nlev, prec=prec, tol=1e-8)
    return dict(kind=kind, shape=shape, nbase=nbase, ni=ni, nlev=nlev, prec=prec, tol=rng.choice([1e-3, 1e-6, 1e-10]),
                warm=rng.random() < 0.3, host=rng.random() < 0.2, table=rng.random() < 0.4)


# ---------------------------------------------------------------------------
@functools.lru_cache(maxsize=6)
def _hierarchy(shape, nbase, ni, nlev):
    """(hierarchy, density function, boundary), kept between preparations."""
    if shape == "uniform":
        return w.uniform_periodic(nbase, ni), w.gaussian_peak, abi.SFM_BC_PERIODIC
    if shape == "nested":
        return w.nested_sphere(nlev, nbase, ni), w.softened_sphere, abi.SFM_BC_SPHERE
    if shape == "sparse":
        return w.small_periodic(nbase, ni, nlev, 5), w.gaussian_peak, abi.SFM_BC_PERIODIC
    if shape == "sparse_sphere":
        return w.small_sphere(nbase, ni, nlev, 5), w.softened_sphere, abi.SFM_BC_SPHERE
    if shape == "cylinder":
        return w.zperiodic_cylinder(nbase, ni, min(nlev, 4)), w.beaded_line, abi.SFM_BC_CYL_ZPERIODIC
    h, fn = w.jeans_cloud(nlev=nlev, nbase=nbase, ni=ni)
    return h, fn, abi.SFM_BC_PERIODIC


@functools.lru_cache(maxsize=3)
def _base_density(shape, nbase, ni, nlev):
    h, fn, _ = _hierarchy(shape, nbase, ni, nlev)
    return w.block_field(h, 2, fn)


def _key(case):
    return case["shape"], case["nbase"], case["ni"], case["nlev"]


def _wave(h, seed, amp):
    """1 + amp * (a seeded wave with the box's period) at every cell, [nb,G,G,G]"""
    rng = np.random.default_rng([seed, 17])
    k, ph = rng.integers(1, 4, 3), rng.uniform(0.0, 2.0 * math.pi, 3)
    c = [torch.from_numpy(v).cuda() for v in w.cell_centres(h, 2)]
    s = [torch.sin((2.0 * math.pi * float(k[d]) / h.box_size) * c[d] + float(ph[d])) for d in range(3)]
    return 1.0 + amp * s[2][:, :, None, None] * s[1][:, None, :, None] * s[0][:, None, None, :]


def _params(case, bc):
    kw = dict(rel_tol=case["tol"], max_outer=30, precision=case["prec"])
    if bc != abi.SFM_BC_PERIODIC:
        kw["zero_mean"] = 0
    if bc == abi.SFM_BC_SPHERE:
        kw["lmax"] = 4
    return abi.default_params(bc, **kw)


def _dense_rho(case, seed):
    n = case["n"]
    rng = np.random.default_rng([seed, 3])
    x = (np.arange(n) + 0.5) / n
    c = rng.uniform(0.3, 0.7, 3)
    r2 = ((x - c[0])[None, None, :] ** 2 + (x - c[1])[None, :, None] ** 2 + (x - c[2])[:, None, None] ** 2)
    return (1.0 + 100.0 * np.exp(-r2 / 0.02)) * (1.0 + 0.1 * rng.standard_normal((n, n, n)))


def prepare(case, seed):
    if case["kind"] == "noalloc":
        rho = torch.from_numpy(_dense_rho(case, seed)).cuda()
        f = abi.load_library().sfm_uniform_solve_noalloc
        f.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_int, ctypes.c_double, ctypes.c_double, ctypes.c_double,
                      ctypes.c_int, ctypes.POINTER(ctypes.c_int), ctypes.POINTER(ctypes.c_double), ctypes.c_void_p]
        f.restype = ctypes.c_int
        return dict(case=case, fn=f, rho=rho, psi=torch.empty_like(rho))
    h, _, bc = _hierarchy(*_key(case))
    if case["kind"] == "link":
        order = np.random.default_rng([seed, 5]).permutation(h.nblocks)
        return dict(case=case, ngb=h.ngb, nlev=h.nlev, periodic=h.periodic,
                    level=torch.from_numpy(h.level[order]).cuda(), ijk=torch.from_numpy(h.ijk[order]).cuda())
    ctx = FMGPoisson(h, params=_params(case, bc))
    if case.get("table"):
        ctx.load_tune_table(TUNED)
    if case["kind"] == "adjoint":
        rng = np.random.default_rng([seed, 7])
        dJ = torch.from_numpy(_base_density(*_key(case))).cuda() * _wave(h, seed, 0.3)
        dJ = dJ * torch.from_numpy(rng.uniform(0.5, 1.5, h.nblocks)).cuda()[:, None, None, None]
        return dict(case=case, ctx=ctx, dJ=dJ.cpu().numpy())
    rho = torch.from_numpy(_base_density(*_key(case))).cuda() * _wave(h, seed, 0.3)
    if case["warm"]:   # the last step's potential: that of a slightly different density
        psi0 = torch.zeros_like(rho)
        prev = rho * _wave(h, seed + 1, 0.02)
        ctx.solve_device(prev.data_ptr(), psi0.data_ptr())
        torch.cuda.synchronize()
    else:
        psi0 = torch.zeros_like(rho)
    if case["host"]:
        return dict(case=case, ctx=ctx, rho=rho.cpu().numpy(), psi0=psi0.cpu().numpy())
    g = torch.zeros((h.nblocks, 3) + rho.shape[1:], dtype=torch.float64, device="cuda")
    return dict(case=case, ctx=ctx, rho=rho, psi0=psi0, psi=torch.zeros_like(rho), g=g)


def run(state):
    kind = state["case"]["kind"]
    if kind == "noalloc":
        c = state["case"]
        state["fn"](state["rho"].data_ptr(), state["psi"].data_ptr(), c["n"], 1.0 / c["n"], 4.0 * math.pi, c["tol"], 200,
                    None, None, torch.cuda.current_stream().cuda_stream)
        return state["psi"] - state["psi"].mean()   # the periodic potential's constant is free
    if kind == "link":
        return link_blocks(state["level"], state["ijk"], state["ngb"], state["periodic"], nlev=state["nlev"],
                           stream=torch.cuda.current_stream().cuda_stream)
    if kind == "adjoint":
        return state["ctx"].adjoint(state["dJ"], allow_unconverged=True)[0]
    if state["case"]["host"]:
        psi, g, _ = state["ctx"].solve(state["rho"], state["psi0"])
        return psi, g
    state["psi"].copy_(state["psi0"])   # the warm start, or zeros: the call solves in place
    torch.cuda.current_stream().synchronize()   # the solve runs on its context's own stream
    state["ctx"].solve_device(state["rho"].data_ptr(), state["psi"].data_ptr(), state["g"].data_ptr())
    return state["psi"], state["g"]


def work(case):
    if case["kind"] == "noalloc":
        n3 = case["n"] ** 3
        # density in, potential out; one red-black sweep's operations per digit asked for
        return {"bytes": 16 * n3, "flops": 10 * n3}
    h, _, _ = _hierarchy(*_key(case))
    cells = h.nblocks * h.ni ** 3
    if case["kind"] == "link":
        return {"bytes": h.nblocks * (16 + 4 * (1 + 8 + 6) + 6), "flops": 0}
    if case["kind"] == "adjoint":
        return {"bytes": 16 * cells, "flops": 10 * cells}
    # density and start in, potential and three components of g out
    return {"bytes": 48 * cells, "flops": 10 * cells}


def tolerance(case):
    if case["kind"] == "link":
        return "exact"
    # Two correct solves stop within rel_tol of the same fixed point; those
    # that run the same iteration with sums in another order agree to the
    # rounding of the doubles that carry the potential, amplified by the
    # differences that form g (measured 1e-13 between the oracle and the
    # mixed path at 1e-10).  The adjoint adds with FP64 atomics, and its
    # Krylov space amplifies their order.
    if case["kind"] == "adjoint":
        return {"rel": 1e-8}
    return {"rel": 1e-9}


def exact(case, seed):
    if case["kind"] == "link":
        h, _, _ = _hierarchy(*_key(case))
        order = np.random.default_rng([seed, 5]).permutation(h.nblocks)
        back = np.empty(h.nblocks + 1, dtype=np.int32)
        back[order] = np.arange(h.nblocks, dtype=np.int32)
        back[-1] = -1
        return back[h.parent[order]], back[h.child[order]], back[h.nbr[order]], h.touch[order]
    if case["kind"] == "noalloc":
        rho, n = _dense_rho(case, seed), case["n"]
        return _fft_solve(rho, n, 1.0 / n)
    if case["kind"] != "solve" or case["shape"] != "uniform" or case["tol"] > 1e-9 or case["nbase"] & (case["nbase"] - 1):
        return None   # a composite hierarchy, or a solve stopped far from its limit: no closed form
    h, _, _ = _hierarchy(*_key(case))
    rho = (torch.from_numpy(_base_density(*_key(case))).cuda() * _wave(h, seed, 0.3)).cpu().numpy()
    ni, n = h.ni, h.ngb[0] * h.ni
    dense = np.empty((n, n, n))
    for b in range(h.nblocks):
        i, j, k = (int(v) * ni for v in h.ijk[b])
        dense[k:k + ni, j:j + ni, i:i + ni] = rho[b, 2:2 + ni, 2:2 + ni, 2:2 + ni]
    hw = float(h.cellwidth[0])
    phi = _fft_solve(dense, n, hw)
    g = np.zeros((h.nblocks, 3) + rho.shape[1:])
    gd = [-(np.roll(phi, -1, ax) - np.roll(phi, 1, ax)) / (2.0 * hw) for ax in (2, 1, 0)]
    for b in range(h.nblocks):
        i, j, k = (int(v) * ni for v in h.ijk[b])
        for d in range(3):
            g[b, d, 2:2 + ni, 2:2 + ni, 2:2 + ni] = gd[d][k:k + ni, j:j + ni, i:i + ni]
    return None, g   # the potential's constant is free; its gradient is not


def _fft_solve(rho, n, hw):
    """The 7-point periodic problem lap(phi) = 4 pi (rho - mean rho), mean phi = 0."""
    k = 2.0 * np.sin(math.pi * np.arange(n) / n)
    lam = -(k[:, None, None] ** 2 + k[None, :, None] ** 2 + k[None, None, :] ** 2) / hw ** 2
    lam[0, 0, 0] = 1.0
    f = np.fft.fftn(4.0 * math.pi * (rho - rho.mean())) / lam
    f[0, 0, 0] = 0.0
    return np.ascontiguousarray(np.fft.ifftn(f).real)
