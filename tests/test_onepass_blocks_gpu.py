"""Exact single-pass kernel where only some tiles leave the range of its
branch-free quotients: values at the edges of the tiles and of the blocks of
columns the prep kernel reports by, in domains that have interior tiles
(extents from 121 x 48 on), and in one member of a batch.  Held to the two-pass
kernels with IEEE division, cell for cell."""
import numpy as np
import pytest

from hicar_b200.advection import AdvOptions, Domain, Options, adv_init
from hicar_b200.batch import Batch
from tests.test_onepass_ranges_gpu import make, run_ieee, same

pytestmark = pytest.mark.gpu

F32 = np.float32
# columns and rows beside the edges of tiles (60, 116; 22, 44), of their planes
# (56, 64, 112, 120; 19, 41, 47) and of the blocks (32; 8)
AT = [(0, 0), (31, 7), (32, 8), (55, 18), (56, 19), (60, 22), (63, 24), (64, 25), (95, 40), (96, 41), (119, 47), (120, 48),
      (127, 46), (140, 30), (175, 66)]


@pytest.mark.parametrize("fct", [True, False])
@pytest.mark.parametrize("wind", ["u", "v", "w"])
@pytest.mark.parametrize("group", range(3))
def test_one_small_wind_at_tile_edges(wind, group, fct):
    case = make("plain", 176, 67, 12)
    q = case.species["qc"]
    rng = np.random.default_rng(group)
    q[...] = (rng.integers(0, 4000, q.shape) * rng.integers(0, 2, q.shape)).astype(np.uint32).view(F32)   # bits that show a lost rounding
    for i, j in AT[group::3]:
        getattr(case, wind)[j, rng.integers(0, case.nz), i] = F32(1e-30)
    same(case, fct=fct)


@pytest.mark.parametrize("fct", [True, False])
@pytest.mark.parametrize("kind", ["subnormal", "tie", "huge", "nonfinite", "negative", "tiny wind", "no wind",
                                  "courant one"])
def test_interior_tiles_equal_ieee_division(kind, fct):
    same(make(kind, 180, 70, 21), fct=fct)


@pytest.mark.parametrize("kind", ["huge", "nonfinite", "tiny wind", "subnormal"])
@pytest.mark.parametrize("fct", [True, False])
def test_one_member_of_a_batch_leaves_the_range(kind, fct):
    cases = [make("plain", 180, 70, 11), make(kind, 180, 70, 11, seed=4), make("plain", 61, 33, 9, seed=5)]
    opts = Options(adv_options=AdvOptions(MPDATA_FCT=fct))
    b, doms = Batch(0), []
    for c in cases:
        d = Domain.from_case(c)
        adv_init(d, opts)
        b.add(d, c.dt)
        doms.append(d)
    for _ in range(3):
        b.step()
    b.sync()
    for c, d in zip(cases, doms):
        want = run_ieee(c, 3, fct)
        b.remove(d)
        for k in want:
            assert np.array_equal(d.fetch(k), want[k], equal_nan=True), k
        d.close()
    b.close()
