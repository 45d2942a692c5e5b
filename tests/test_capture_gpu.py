"""Steps captured in a CUDA graph from a caller's stream after one plain step:
the replays advance the fields as plain steps do."""
import ctypes as C

import numpy as np
import pytest
import torch

from hicar_b200 import _lib as L
from hicar_b200 import synth
from hicar_b200.advection import AdvOptions, Domain, Options, PhysicsOptions, TimeOptions, adv_init, step

pytestmark = pytest.mark.gpu


def domain(case, opts, path):
    d = Domain.from_case(case)
    adv_init(d, opts)
    d.set_path(path)
    for k, v in case.species.items():
        d.set_forcing(k, (v * np.float32(1.1)).astype(np.float32), (v * np.float32(1e-4)).astype(np.float32))
    return d


@pytest.mark.parametrize("scheme", ["exact", "fast", "standard"])
def test_replayed_steps_equal_plain_ones(scheme):
    case = synth.config2(seed=8, nx=140, ny=60, nz=11)
    case.species = {k: case.species[k] for k in ("qv", "qc", "theta")}
    opts = Options()
    if scheme == "standard":
        opts = Options(physics=PhysicsOptions(advection=1), adv_options=AdvOptions(h_order=3, v_order=3, flux_corr=1),
                       time_options=TimeOptions(RK3=False))
    path = 3 if scheme == "fast" else 0
    want = domain(case, opts, path)
    for _ in range(5):
        step(want, opts, case.dt, enforce_limits=True)
    d = domain(case, opts, path)
    s = torch.cuda.Stream()
    L.check(L.load().icar_adv_set_stream(d.handle, C.c_void_p(s.cuda_stream)), d.handle)
    step(d, opts, case.dt, enforce_limits=True)
    d.sync()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s, capture_error_mode="thread_local"):
        for _ in range(2):
            step(d, opts, case.dt, enforce_limits=True)
    with torch.cuda.stream(s):
        g.replay()
        g.replay()
    s.synchronize()
    for k in case.species:
        assert np.array_equal(d.fetch(k), want.fetch(k)), k
    d.close()
    want.close()
