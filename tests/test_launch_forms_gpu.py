"""One domain's steps through every form of the single-pass launch: all species
in one launch, each species in a launch of its own (which cuts the columns into
other level ranges), the host-memory step (a species per launch), and a batch
beside other members.  The fields have to be equal bit for bit, in exact and in
fast arithmetic."""
import numpy as np
import pytest

from hicar_b200 import synth
from hicar_b200.advection import AdvOptions, Domain, Options, adv_init, advect, step_host
from hicar_b200.batch import Batch

pytestmark = pytest.mark.gpu

STEPS = 3


def domain(case, opts, path):
    d = Domain.from_case(case)
    adv_init(d, opts)
    d.set_path(path)
    return d


@pytest.mark.parametrize("fct", [True, False])
@pytest.mark.parametrize("path", [2, 3])
@pytest.mark.parametrize("nx,ny,nz,names", [(180, 70, 21, ("qv", "qc", "theta")),          # interior tiles, short launches
                                            (130, 95, 47, ("qv", "qc", "theta", "nr", "qr", "qs", "qi")),
                                            (250, 210, 23, ("qv", "qc", "theta")),         # 150 tiles: a wave and two
                                            (61, 33, 9, ("qc", "nr"))])
def test_every_form_of_the_launch_gives_the_same_fields(nx, ny, nz, names, path, fct):
    case = synth.config2(seed=nx, nx=nx, ny=ny, nz=nz)
    case.species = {k: case.species[k] for k in names}
    opts = Options(adv_options=AdvOptions(MPDATA_FCT=fct))
    d = domain(case, opts, path)
    for _ in range(STEPS):
        advect(d, opts, case.dt)
    want = {k: d.fetch(k).copy() for k in names}
    d.close()
    # a species at a time
    for k in names:
        one = case.copy()
        one.species = {k: case.species[k]}
        d = domain(one, opts, path)
        for _ in range(STEPS):
            advect(d, opts, case.dt)
        assert np.array_equal(d.fetch(k), want[k]), k
        d.close()
    # host-memory steps
    d = domain(case, opts, path)
    host = {k: v.copy() for k, v in case.species.items()}
    for _ in range(STEPS):
        step_host(d, opts, case.dt, host, host)
    for k in names:
        assert np.array_equal(host[k], want[k]), k
    d.close()
    # a batch, alone and beside a larger member
    for others in ([], [synth.config2(seed=1, nx=200, ny=150, nz=30)]):
        b, doms = Batch(0), []
        b.set_path(path)
        for c in [case] + others:
            m = domain(c, opts, path)
            b.add(m, c.dt)
            doms.append(m)
        for _ in range(STEPS):
            b.step()
        b.sync()
        b.remove(doms[0])
        for k in names:
            assert np.array_equal(doms[0].fetch(k), want[k]), k
        for m in doms[1:]:
            b.remove(m)
        for m in doms:
            m.close()
        b.close()
