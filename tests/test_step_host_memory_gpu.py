"""icar_adv_step_host where the device has room for the step but not for its
staging buffers, in a process of its own (no memory kept from other tests):
the staging gives way to what the step and later calls need."""
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu
ROOT = Path(__file__).resolve().parents[1]

PROGRAM = """
import ctypes as C, sys
import numpy as np, torch
from hicar_b200 import _lib as L, synth
from hicar_b200.advection import AdvOptions, Domain, Options, PhysicsOptions, TimeOptions, adv_init, step, step_host
room = int(sys.argv[1])          # fields of the domain left free
case = synth.config2(seed=2, nx=508, ny=512, nz=40)
case.species = {k: case.species[k] for k in ("qv", "qc", "theta")}
opts = Options(physics=PhysicsOptions(advection=1), adv_options=AdvOptions(h_order=3, v_order=3),
               time_options=TimeOptions(RK3=True))
def make():
    d = Domain.from_case(case)
    adv_init(d, opts)
    d.sync()
    return d
d = make()
field = 4 * 512 * 512 * 40
free, _ = torch.cuda.mem_get_info()
fill = torch.empty(free - room * field - (96 << 20), dtype=torch.uint8, device="cuda")
host = {k: v.copy() for k, v in case.species.items()}
for _ in range(2):
    step_host(d, opts, case.dt, host, host)
del fill
torch.cuda.empty_cache()
e = make()
for _ in range(2):
    step(e, opts, case.dt)
for k in host:
    assert np.array_equal(host[k], e.fetch(k)), k
print("ok")
"""


@pytest.mark.parametrize("room", [7, 8, 30])   # beside 96 MB: the step needs 8 fields of 42 MB, the staging 4 more
def test_step_runs_without_room_for_staging(room):
    r = subprocess.run([sys.executable, "-c", PROGRAM, str(room)], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "ok" in r.stdout, r.stderr[-2000:]
