"""Calls whose time has to stay near that of a neighbouring call: extents that
leave threads without a cell, values that take the long way."""
import time

import numpy as np
import pytest
import torch

from hicar_b200 import synth
from hicar_b200.advection import Domain, Options, Parameters, advect, balance_uvw
from hicar_b200.batch import Batch

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


def test_batch_forgets_a_step_outside_the_exact_range():
    """A wind too small for the branch-free quotients sends a member's tiles to
    IEEE division; once it is gone so is its cost, without new tables."""
    opts = Options()
    d, dt = device_domain(180, 160, 30, opts, ("qv", "theta", "qc"))
    b = Batch(0)
    b.add(d, dt)
    v = d.download(["v"])["v"]
    small = v.copy()
    small[...] = 1e-30
    for _ in range(4):
        b.step()
    t = [microseconds(b.step, b.sync, n=10)]
    for a in (small, v):
        d.upload("v", a)
        b.step()
        b.step()
        t.append(microseconds(b.step, b.sync, n=10))
    b.remove(d)
    b.close()
    d.close()
    assert t[1] > 1.5 * t[0] and t[2] < 1.2 * t[0], t


def test_one_wind_outside_the_exact_range_costs_its_tiles_only():
    opts = Options()
    names = ("qv", "theta", "qc", "qr", "qs", "qi")
    t = []
    for change in (None, lambda f: f["u"].__setitem__((20, 3, 30), 1e-30)):
        d, dt = device_domain(384, 384, 30, opts, names, change)
        t.append(microseconds(lambda: advect(d, opts, dt), d.sync, n=10))
        d.close()
    assert t[1] < 1.5 * t[0], t


@pytest.mark.parametrize("path", [0, 3])
def test_a_launch_just_above_a_wave_costs_little_more_than_the_wave(path):
    """Six species of 96 x 250 are 144 column tiles, one wave of the 148 SMs;
    seven are 168."""
    opts = Options()
    names = ("qv", "theta", "qc", "qr", "qs", "qi", "qg")
    t = []
    for n in (6, 7):
        d, dt = device_domain(96, 250, 35, opts, names[:n])
        d.set_path(path)
        t.append(microseconds(lambda: advect(d, opts, dt), d.sync, n=20))
        d.close()
    assert t[1] < 1.38 * t[0], t   # a sixth more tiles; with a second wave of whole columns 1.42 and 1.47
