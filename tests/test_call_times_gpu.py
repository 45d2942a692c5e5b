"""Calls whose time has to stay near that of a neighbouring call: extents that
leave threads without a cell, values that take the long way."""
import time

import numpy as np
import pytest
import torch

from hicar_b200 import synth
from hicar_b200.advection import Domain, Options, Parameters, balance_uvw

pytestmark = pytest.mark.gpu


def device_domain(nx, ny, nz, opts, species=("qv",), change=None):
    f, dt = synth.device_member(nx, ny, nz, 3, species=species, U=10.0)
    if change:
        change(f)
    d = Domain.create_on_device(f, nx, ny, nz, 4000.0, opts)
    d._device_fields = None
    return d, dt


def microseconds(call, sync, n=40, repeats=9):
    """Least time of a call among n queued one after the other."""
    best = []
    for _ in range(repeats):
        call()
        sync()
        t = time.perf_counter()
        for _ in range(n):
            call()
        sync()
        best.append((time.perf_counter() - t) / n * 1e6)
    return min(best)


def test_balance_of_ragged_extents_costs_what_the_aligned_ones_around_it_do():
    opts = Options(parameters=Parameters(advect_density=True))
    t = []
    for n in (100, 128):   # 100: the last tiles have columns outside the domain
        d, _ = device_domain(n, n, 40, opts)
        t.append(microseconds(lambda: balance_uvw(d, opts), d.sync))
        d.close()
    assert t[0] < 1.15 * t[1], t
