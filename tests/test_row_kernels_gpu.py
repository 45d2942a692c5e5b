"""The per-row kernels of a step (boundary relaxation, per-step fields,
clipping, stable time step) at every remainder of their four-value groups and
four-level groups, cell for cell against the oracle."""
import numpy as np
import pytest

from hicar_b200 import synth
from hicar_b200.advection import (Domain, Options, Parameters, TimeOptions, adv_init, advect, compute_dt)

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("den", [0, 1])
@pytest.mark.parametrize("nx,ny,nz", [(60, 24, 3), (61, 23, 4), (62, 25, 5), (63, 31, 9), (5, 4, 3)])
def test_rows_match_oracle(oracle_lib, nx, ny, nz, den):
    O = oracle_lib
    case = synth.config2(seed=nx + den, nx=nx, ny=ny, nz=nz)
    case.species = {k: case.species[k] for k in ("qc", "qv")}
    rng = np.random.default_rng(nx)
    q = case.species["qc"]
    q[...] = (rng.standard_normal(q.shape) * 1e-4).astype(np.float32)
    opts = Options(parameters=Parameters(advect_density=bool(den)), time_options=TimeOptions(cfl_strictness=3))
    # boundary relaxation, then the step on its per-step fields
    forcing = {k: ((v * np.float32(1.1)).astype(np.float32), (v * np.float32(1e-4)).astype(np.float32))
               for k, v in case.species.items()}
    flt = O.init_relax_filters(nx, ny, 2)
    ref = O.run_steps(case, O.make_opts(advect_density=den), case.dt, 2, forcing=forcing, filter2d=flt)
    d = Domain.from_case(case)
    adv_init(d, opts)
    for k, (fh, dq) in forcing.items():
        d.set_forcing(k, fh, dq)
    for _ in range(2):
        d.apply_forcing(case.dt)
        advect(d, opts, case.dt)
    for k in ref:
        assert np.array_equal(d.fetch(k), ref[k]), k
    # clipping
    d.enforce_limits()
    for k in ref:
        want = ref[k].copy()
        O.enforce_limits(want)
        assert np.array_equal(d.fetch(k), want), k
    # the stable time step
    dz = np.asarray(case.dz_levels, np.float32)
    want, small = O.compute_dt(case, 2, dz, 0.9, 3)
    assert not small and compute_dt(d, opts, dz) == want
    d.close()
