"""The stable time step of winds that hold NaN: NaN for a wind that is NaN
throughout, whichever it is; a NaN among other values is skipped."""
import numpy as np
import pytest

from hicar_b200 import synth
from hicar_b200.advection import Domain, Options, TimeOptions, adv_init, compute_dt

pytestmark = pytest.mark.gpu


def domain(strictness):
    case = synth.config2(seed=5, nx=61, ny=23, nz=9)
    case.species = {"qv": case.species["qv"]}
    d = Domain.from_case(case)
    opts = Options(time_options=TimeOptions(cfl_strictness=strictness, cfl_reduction_factor=900.0))
    adv_init(d, opts)
    return case, d, opts, np.full(case.nz, 500.0, np.float32)


@pytest.mark.parametrize("strictness", [1, 2, 3, 4, 5])
@pytest.mark.parametrize("wind", ["u", "v", "w"])
def test_time_step_of_nan_winds(wind, strictness):
    case, d, opts, dz = domain(strictness)
    sound = compute_dt(d, opts, dz)
    a = getattr(case, wind).copy()
    a[1, 2, 0] = a[11, 4, 31] = a[-1, -1, -1] = 0.0
    d.upload(wind, a)
    without = compute_dt(d, opts, dz)          # the same winds with zeros in three places
    a[1, 2, 0] = a[11, 4, 31] = a[-1, -1, -1] = np.nan
    d.upload(wind, a)
    assert np.isfinite(sound) and compute_dt(d, opts, dz) == without
    d.upload(wind, np.full_like(a, np.nan))
    assert np.isnan(compute_dt(d, opts, dz))
    assert np.isinf(compute_dt(d, opts, dz, use_density=True))
    d.close()
