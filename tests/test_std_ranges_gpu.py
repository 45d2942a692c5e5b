"""Standard-scheme kernels outside the values their branch-free quotients are
formed for, and at the edges of their range: equal to the oracle cell for
cell, NaN for NaN."""
import numpy as np
import pytest

from tests.test_onepass_ranges_gpu import F32, make
from tests.test_parity_gpu import gpu_run
from tests.test_std_fused_gpu import std_options

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("h,v,fc,rk3", [(5, 3, 1, 1), (3, 5, 0, 0), (1, 1, 1, 0)])
@pytest.mark.parametrize("kind", ["subnormal", "tie", "huge", "overflow", "nonfinite", "negative", "no wind",
                                  "thin air"])
def test_std_kernels_match_oracle(oracle_lib, kind, h, v, fc, rk3):
    O = oracle_lib
    case = make(kind)
    if kind == "overflow":             # finite values whose fluxes are not
        q = case.species["nr"]
        q[tuple(np.random.default_rng(2).integers(0, n, 6) for n in q.shape)] = F32(3e38)
    if kind == "thin air":             # J*rho below the range of the exact quotients
        case.density[...] = F32(1e-8)
    den = int(kind == "thin air")
    with np.errstate(all="ignore"):
        ref = O.run_steps(case, O.make_opts(advection=1, h_order=h, v_order=v, flux_corr=fc, rk3=rk3,
                                            advect_density=den), case.dt, 2)
    out = gpu_run(case, std_options(h, v, fc, rk3, den=bool(den)), 2)
    for k in ref:
        assert np.array_equal(out[k], ref[k], equal_nan=True), (k, int((out[k] != ref[k]).sum()))
