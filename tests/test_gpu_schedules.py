"""The two kernels of the right-hand side, which a step takes by the level's
size and by how many evolutions are stepped beside it, give the same bits:
every variant of the physics alone (a block per tile) and beside others (a
cell per tile), queued side by side and in fused launches."""
import numpy as np
import pytest

from parity_util import C1, field_list, params

pytestmark = pytest.mark.gpu

BESIDE = 48  # other evolutions, small enough not to matter
GD2 = dict(shift="Gammadriver2", drivercsi=0.75, drivereta=2.0)
FIELD = dict(idata="minkowski", ilapse="one", mattertype="scalar", scalarpotential="phi2", scalar_mass=0.5, scalardiss=0.02)
BOX = dict(nrtotal=24, nztotal=24, dr0=0.25, dz0=0.25, Nb=1, Nl1=1, Nrbox1=16, Nzbox1=16, zbox1=2.0)

VARIANTS = {
    "vacuum": {},
    "shift": GD2,
    "scalar": FIELD,
    "shift_scalar": dict(FIELD, **GD2),
    "centred_advection": dict(GD2, shiftadvect=0),
    "centred_advection_scalar": dict(FIELD, shiftadvect=0, **GD2),
    "driver0": dict(shift="Gammadriver0", drivercsi=0.1, dr0=0.25, dz0=0.25, eqsym=0),
    "driver1": dict(GD2, shift="Gammadriver1"),
    "driver1_D0": dict(GD2, shift="Gammadriver1", driverD0=1),
    "driver1_advected": dict(GD2, shift="Gammadriver1", driveradv=1),
    "driver2_advected": dict(GD2, driveradv=1),
    "driver2_centred": dict(GD2, driveradv=1, shiftadvect=0),
    "shock1": dict(GD2, shift="Gammadrivershock1"),
    "shock2": dict(GD2, shift="Gammadrivershock2", driverD0=1),
    "static": dict(boundtype="static"),
    "flat": dict(GD2, boundtype="flat"),
    "no_equator": dict(GD2, eqsym=0),
    "no_equator_scalar": dict(FIELD, eqsym=0),
    "four_ghosts": dict(GD2, ghost=4),
    "harmonic": dict(slicing="harmonic", gauge_f=1.0),
    "order_two": dict(order="two", integrator="icn", icniter=3),
    "order_two_all": dict(FIELD, order="two", eqsym=0, **GD2),
    "maximal": dict(maximalevery=1, we_maxiter=60, nl0=0),
    "maximal_slicing": dict(slicing="maximal", ilapse="maximal", we_maxiter=60, nl0=0),
    "boxes": dict(GD2, **BOX),
    "boxes_scalar": dict(FIELD, **BOX),
    "boxes_maximal": dict(maximalevery=1, we_maxiter=60, **BOX),
}


def make(cfg):
    from ollin.gpu import Evolution
    e = Evolution(params(cfg))
    e.initial_data()
    e.initialize()
    if is_maximal(cfg):
        e.maximal_slicing()
    return e


def is_maximal(cfg):
    return bool(cfg.get("maximalevery")) or cfg.get("slicing") == "maximal"


@pytest.fixture(scope="module")
def others():
    es = [make(dict(C1, nrtotal=16, nztotal=16, nl0=0, idata="minkowski", ilapse="one")) for _ in range(BESIDE)]
    yield es
    for e in es:
        e.close()


@pytest.mark.parametrize("name", VARIANTS)
def test_a_step_is_the_same_whatever_runs_beside_it(name, others):
    from ollin.gpu import step_fused, step_many
    cfg = dict(dict(C1, nrtotal=42, nztotal=37, nl0=1), **VARIANTS[name])
    alone, many, fused, mixed = [make(cfg) for _ in range(4)]
    ways = [lambda e: e.step(), lambda e: step_many([e] + others), lambda e: step_fused([e] + others)]
    for step in range(3):
        ways[0](alone)
        ways[1](many)
        ways[2](fused)
        ways[(step + 1) % 3](mixed)
        if is_maximal(cfg):
            for e in (alone, many, fused, mixed):
                e.maximal_slicing()
        for lev in alone.levels():
            for nm in field_list(cfg):
                a = alone.download(lev, nm)
                for way, e in (("many", many), ("fused", fused), ("mixed", mixed)):
                    assert np.array_equal(a, e.download(lev, nm)), (step, way, lev, nm)
    for e in (alone, many, fused, mixed):
        e.close()


# members of one group of fused launches: grids of both kernels alone (288 and
# 432 tiles, 619 and 855), and with few others and many, so that a cell takes one
# tile and several
@pytest.mark.parametrize("kind", ["vacuum", "shift", "scalar", "order_two"])
@pytest.mark.parametrize("count", [1, 12])
def test_fused_steps_of_large_grids_equal_single_steps(kind, count):
    from ollin.gpu import step_fused
    sizes = [(96, 96), (144, 96), (165, 120), (201, 136)]
    cfgs = [dict(dict(C1, nrtotal=nr, nztotal=nz, nl0=0, dr0=16.0 / nr, dz0=16.0 / nr), **VARIANTS[kind]) for nr, nz in sizes]
    alone = [make(c) for c in cfgs]
    batch = [make(c) for c in cfgs for _ in range(count)]
    for step in range(3):
        t = [e.step() for e in alone]
        if step == 1:
            assert [e.step() for e in batch][::count] == t
        else:
            assert step_fused(batch)[::count] == t
    for k, (cfg, a) in enumerate(zip(cfgs, alone)):
        for nm in field_list(cfg):
            want = a.download(0, nm)
            for e in batch[k * count:(k + 1) * count]:
                assert np.array_equal(want, e.download(0, nm)), (sizes[k], nm)
    for e in alone + batch:
        e.close()
