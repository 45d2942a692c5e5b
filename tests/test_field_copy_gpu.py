"""Field copies between a caller's contiguous device memory and the handle's
pitched rows: exact, whatever the row length and the caller's alignment, and
nothing outside the caller's array is written."""
import ctypes as C

import numpy as np
import pytest
import torch

from hicar_b200 import _lib as L
from hicar_b200 import synth
from hicar_b200.advection import Domain, Options, adv_init

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shift", [0, 1, 4])
@pytest.mark.parametrize("nx,ny,nz", [(3, 3, 3), (7, 5, 4), (64, 23, 9), (65, 17, 3), (1027, 6, 3), (4100, 3, 3)])
def test_device_field_round_trip(nx, ny, nz, shift):
    case = synth.config2(seed=1, nx=nx, ny=ny, nz=nz)
    case.species = {k: case.species[k] for k in ("qc", "nr")}
    d = Domain.from_case(case)
    adv_init(d, Options())
    lib = L.load()
    g = torch.Generator(device="cuda").manual_seed(nx + shift)
    for fid, ex, ey in ((L.SPECIES_IDS["qc"], nx, ny), (L.F_U, nx + 1, ny), (L.F_V, nx, ny + 1)):
        n = ex * nz * ey
        src = torch.randn(n + 16, generator=g, device="cuda")
        out = torch.full((n + 16,), 7.0, device="cuda")
        torch.cuda.synchronize()
        L.check(lib.icar_adv_set_field_device(d.handle, fid, C.c_void_p(src.data_ptr() + 4 * shift)),
                d.handle)
        L.check(lib.icar_adv_get_field_device(d.handle, fid, C.c_void_p(out.data_ptr() + 4 * shift)),
                d.handle)
        host = np.empty((ey, nz, ex), np.float32)
        L.check(lib.icar_adv_get_field(d.handle, fid, host.ctypes.data_as(C.c_void_p), None), d.handle)
        d.sync()
        want = torch.full_like(out, 7.0)
        want[shift:shift + n] = src[shift:shift + n]
        assert torch.equal(out, want)
        assert np.array_equal(host.ravel(), src[shift:shift + n].cpu().numpy())
    d.close()
