"""Exact single-pass MPDATA kernel outside the values its branch-free
quotients are formed for, and at the edges of their range.

The reference here is the step on caller-owned memory, whose two-pass kernels
divide with the compiler's IEEE division everywhere (themselves held to the
oracle elsewhere); the results have to be equal cell for cell, NaN for NaN.
"""
import ctypes as C

import numpy as np
import pytest
import torch

from hicar_b200 import _lib as L
from hicar_b200 import synth
from hicar_b200.advection import Domain, Options, AdvOptions, adv_init, advect

pytestmark = pytest.mark.gpu

F32 = np.float32


def run(case, path, nsteps, fct=True):
    d = Domain.from_case(case)
    opts = Options(adv_options=AdvOptions(MPDATA_FCT=fct))
    adv_init(d, opts)
    d.set_path(path)
    for _ in range(nsteps):
        advect(d, opts, case.dt)
    out = {k: d.fetch(k).copy() for k in case.species}
    d.sync()
    d.close()
    return out


def run_ieee(case, nsteps, fct=True):
    """The same steps through icar_adv_advect_noalloc."""
    P = (case.nx + 4) // 4 * 4

    def pitched(a):
        t = torch.zeros((a.shape[0], a.shape[1], P), device="cuda")
        t[:, :, :a.shape[2]] = torch.from_numpy(np.ascontiguousarray(a))
        return t
    met = ("u", "v", "w", "density", "jacobian", "jacobian_u", "jacobian_v", "jacobian_w", "advection_dz")
    fields = {k: pitched(getattr(case, k)) for k in met}
    cur = {k: pitched(v) for k, v in case.species.items()}
    for _ in range(nsteps):
        nxt = {k: torch.zeros_like(v) for k, v in cur.items()}
        a = L.NoallocArgs()
        a.nx, a.ny, a.nz, a.dx, a.dt, a.mpdata_fct, a.n_species = case.nx, case.ny, case.nz, case.dx, case.dt, int(fct), len(cur)
        for k in met:
            setattr(a, k, fields[k].data_ptr())
        for s, k in enumerate(cur):
            a.q_in[s], a.q_out[s] = cur[k].data_ptr(), nxt[k].data_ptr()
        torch.cuda.synchronize()
        assert L.load().icar_adv_advect_noalloc(C.byref(a)) == L.OK
        torch.cuda.synchronize()
        cur = nxt
    return {k: v[:, :, :case.nx].cpu().numpy() for k, v in cur.items()}


def same(case, nsteps=2, fct=True):
    a, b = run(case, 2, nsteps, fct), run_ieee(case, nsteps, fct)
    for k in b:
        assert np.array_equal(a[k], b[k], equal_nan=True), (k, int((a[k] != b[k]).sum()))


def make(kind, nx=70, ny=47, nz=9, seed=3):
    case = synth.config2(seed=seed, nx=nx, ny=ny, nz=nz)
    case.species = {k: case.species[k] for k in ("qc", "nr", "theta")}
    rng = np.random.default_rng(seed)
    q = case.species["qc"]
    at = tuple(rng.integers(0, n, 6) for n in q.shape)
    if kind == "subnormal":            # tails down to the smallest subnormals
        case.species["qc"] = (rng.integers(0, 4000, q.shape) * rng.integers(0, 2, q.shape)).astype(np.uint32).view(F32)
        case.species["nr"] = (case.species["nr"] * F32(1e-38)).astype(F32)
    elif kind == "tie":                # J*rho = 1, dz*J*rho an even integer: halfway quotients
        for f in ("density", "jacobian", "jacobian_u", "jacobian_v", "jacobian_w"):
            getattr(case, f)[:] = 1
        case.advection_dz[:] = 500
        case.species["qc"] = (rng.integers(0, 4000, q.shape)).astype(np.uint32).view(F32)
    elif kind == "huge":
        case.species["nr"][at] = 3e20
    elif kind == "nonfinite":
        case.species["nr"][at] = np.inf
        q[at] = np.nan
    elif kind == "negative":           # sums of neighbours that cancel
        case.species["qc"] = (1e-9 * rng.standard_normal(q.shape)).astype(F32)
    elif kind == "tiny wind":
        case.v[...] = (1e-30 * rng.standard_normal(case.v.shape)).astype(F32)
    elif kind == "no wind":
        case.u[...] = case.v[...] = case.w[...] = 0
    elif kind == "courant one":        # faces whose Courant number is exactly 1
        for f in ("density", "jacobian", "jacobian_u", "jacobian_v", "jacobian_w", "advection_dz"):
            getattr(case, f)[:] = 1
        case.u[...], case.v[...], case.w[...] = case.dx / case.dt, 0, 0
    return case


@pytest.mark.parametrize("fct", [True, False])
@pytest.mark.parametrize("kind", ["subnormal", "tie", "huge", "nonfinite", "negative", "tiny wind", "no wind",
                                  "courant one"])
def test_exact_kernel_equals_ieee_division(kind, fct):
    same(make(kind), fct=fct)


@pytest.mark.parametrize("nx,ny,nz", [(64, 21, 3), (65, 22, 4), (61, 23, 5), (120, 44, 6), (121, 45, 12), (176, 67, 21)])
def test_tile_and_level_edges(nx, ny, nz):
    """Extents around the 22-row tiles, the column tiles' 64/120/176 edges and the shortest columns."""
    same(make("plain", nx, ny, nz))
