"""A grid that an engine refuses half-way leaves it with the grid, the near-wall table and the
launch it stepped with: its flow goes on bit for bit like that of an engine that never saw the
refused one.  A closure refuses lattices above 1024 cells a side, after the new lattice's
near-wall table has been built; a row too long for the step's ring is refused by every
precision."""
import numpy as np
import pytest

from aerosim_b200 import AerosimError, meshes, sgs
from aerosim_b200 import _native as N

pytestmark = pytest.mark.gpu

SMALL = (64, 24, 26)
CFG = {"uInletLattice": 0.06, "nuLattice": 0.004, "smagorinskyCs": 0.1}


def _voxelize(e, dims, precision, body=None, reset=True):
    h = dims[1] * 0.1
    e.voxelize(body or meshes.uv_sphere(0.6, 20, 16), None, {"length": dims[0] * 0.1, "width": dims[2] * 0.1, "height": h},
               dict(zip(("nx", "ny", "nz"), dims)), dict(CFG, precision=precision), reset_flow=reset)


def _pair(cls, precision, closure):
    made = []
    for _ in range(2):
        e = cls(0)
        if closure:
            e.set_sgs_mlp(sgs.init_params(3))
        _voxelize(e, SMALL, precision)
        e.step(5)
        made.append(e)
    return made


def _same(a, b):
    ga, gb = a.read_voxel_grid(), b.read_voxel_grid()
    assert (ga.nx, ga.ny, ga.nz, ga.dx) == (gb.nx, gb.ny, gb.nz, gb.dx)
    assert np.array_equal(ga.cellFlags, gb.cellFlags) and np.array_equal(ga.boundaryQValues, gb.boundaryQValues)
    assert np.array_equal(a.read_populations().view(np.uint32), b.read_populations().view(np.uint32))
    assert a.read_forces().fx == b.read_forces().fx and a.mass_stats() == b.mass_stats()


# a side above 1024 with the closure (f16s: its rows fit the ring), a row longer than two slots
REFUSED = [("f16s", True, (1040, 8, 8)), ("f32", True, (40, 1030, 6)), ("f32", False, (1600, 6, 6)),
           ("f64", False, (900, 6, 6))]


@pytest.mark.parametrize("reset", [True, False])
@pytest.mark.parametrize("precision,closure,dims", REFUSED, ids=lambda v: str(v))
def test_refused_grid_leaves_the_engine_as_it_was(gpu_engine_cls, precision, closure, dims, reset):
    e, untouched = _pair(gpu_engine_cls, precision, closure)
    for _ in range(2):
        with pytest.raises(AerosimError):
            _voxelize(e, dims, precision, meshes.box(0.3, 0.3, 0.3, 1), reset)
        _same(e, untouched)
        e.step(3), untouched.step(3)
        _same(e, untouched)
    # and a grid that is taken: as in a fresh engine
    fresh = gpu_engine_cls(0)
    if closure:
        fresh.set_sgs_mlp(sgs.init_params(3))
    for x in (e, fresh):
        _voxelize(x, (48, 20, 22), precision)
        x.step(4)
    _same(e, fresh)
    for x in (e, untouched, fresh):
        x.close()


@pytest.mark.parametrize("then", ["back", "other lattice"])
def test_precision_that_does_not_fit_leaves_no_flow(gpu_engine_cls, then):
    """Rows of 2000 cells fit the ring in 16 bits, not in 32: the engine must not step 32-bit
    populations with the launch of the 16-bit ones."""
    e, fresh = gpu_engine_cls(0), gpu_engine_cls(0)
    _voxelize(e, (2000, 6, 6), "f16s")
    e.step(2)
    with pytest.raises(AerosimError) as err:
        e.update_config({"precision": "f32"})
    assert err.value.code == N.ERR_ARG
    for call in (lambda: e.step(1), e.reset_flow, e.read_populations):
        with pytest.raises(AerosimError) as err:
            call()
        assert err.value.code == N.ERR_STATE
    if then == "back":
        e.update_config({"precision": "f16s"})
        _voxelize(fresh, (2000, 6, 6), "f16s")
    else:
        for x in (e, fresh):
            _voxelize(x, SMALL, "f32")
    e.step(4), fresh.step(4)
    _same(e, fresh)
    e.close(), fresh.close()


@pytest.mark.parametrize("dims", [(1040, 8, 8), (40, 6, 1030)], ids=str)
def test_refused_closure_leaves_the_engine_as_it_was(gpu_engine_cls, dims):
    """Wall distances are refused above 1024 cells a side: no closure then, and the launch
    without one goes on."""
    e, untouched = gpu_engine_cls(0), gpu_engine_cls(0)
    for x in (e, untouched):
        _voxelize(x, dims, "f32")
        x.step(3)
    for _ in range(2):
        with pytest.raises(AerosimError):
            e.set_sgs_mlp(sgs.init_params(3))
        e.step(3), untouched.step(3)
        _same(e, untouched)
    # a lattice that allows one: none is set
    for x in (e, untouched):
        _voxelize(x, SMALL, "f32")
        x.step(3)
    _same(e, untouched)
    e.close(), untouched.close()
