"""Device field copies at the sizes where a block's share of rows changes: a value
per thread on small fields, eight (or four 16-byte ones) on large ones, rows
longer than a block's share."""
import ctypes as C

import pytest
import torch

from hicar_b200 import _lib as L
from hicar_b200 import synth
from hicar_b200.advection import Domain, Options

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,nz", [(3, 3, 3), (16, 16, 10), (35, 25, 37), (67, 60, 19), (68, 60, 19), (125, 61, 40),
                                      (128, 63, 38), (259, 40, 60), (260, 74, 64), (2501, 9, 5), (8200, 6, 4)])
def test_set_then_get_returns_the_field(nx, ny, nz):
    f, _ = synth.device_member(nx, ny, nz, 1, species=("qv",), dz=3000.0)
    d = Domain.create_on_device(f, nx, ny, nz, 4000.0, Options())
    d._device_fields = None
    lib = L.load()
    for name, fid, shape in (("qv", L.SPECIES_IDS["qv"], (ny, nz, nx)), ("u", L.F_U, (ny, nz, nx + 1)), ("v", L.F_V, (ny + 1, nz, nx))):
        src = torch.randn(shape, device="cuda")
        got = torch.full((src.numel() + 8,), 7.0, device="cuda")
        torch.cuda.synchronize()
        L.check(lib.icar_adv_set_field_device(d.handle, fid, C.c_void_p(src.data_ptr())), d.handle)
        L.check(lib.icar_adv_get_field_device(d.handle, fid, C.c_void_p(got.data_ptr() + 16)), d.handle)
        d.sync()
        assert torch.equal(got[4:-4].view(shape), src), name
        assert bool((got[:4] == 7).all()) and bool((got[-4:] == 7).all())
    d.close()
