"""A batch whose engines get another body between steps: each instance steps with the near-wall
cells of its current grid (also from a captured graph), like the same engine stepped alone; an
engine on another lattice or in another precision makes the batch refuse."""
import numpy as np
import pytest

from aerosim_b200 import AerosimError, LBMBatch, meshes
from aerosim_b200 import _native as N

pytestmark = pytest.mark.gpu

EVEN, ODD = [(64, 24, 24), (96, 32, 24)], [(65, 24, 24), (96, 32, 24)]


def _voxelize(e, dims, radius, reset=True, precision="f32"):
    h = dims[1] * 0.1
    e.voxelize(meshes.uv_sphere(radius, 24, 20), None, {"length": dims[0] * 0.1, "width": dims[2] * 0.1, "height": h},
               dict(zip(("nx", "ny", "nz"), dims)),
               {"uInletLattice": 0.06, "nuLattice": 0.004, "smagorinskyCs": 0.1, "precision": precision}, reset_flow=reset)


@pytest.mark.parametrize("dims", [EVEN, ODD], ids=["even", "odd"])
@pytest.mark.parametrize("graph_steps", [1, 4])
def test_bodies_change_between_steps(gpu_engine_cls, dims, graph_steps):
    made = [[gpu_engine_cls(0) for _ in dims] for _ in range(2)]
    for es in made:
        for e, d in zip(es, dims):
            _voxelize(e, d, 0.5)
    batch = LBMBatch(made[0])
    batch.set_tuning(2, 1, graph_steps, 512)
    # a larger body, a much smaller one, the first one again: in one instance, then the other
    for k, radius in ((None, 0), (0, 0.8), (1, 0.25), (0, 0.3), (1, 0.5)):
        if k is not None:
            for es in made:
                _voxelize(es[k], dims[k], radius, reset=False)
        batch.step(9)
        for e in made[1]:
            e.step(9)
        for a, b in zip(*made):
            solid = np.tile(b.read_voxel_grid().cellFlags == 1, 19)
            fa, fb = a.read_populations().astype(np.float64), b.read_populations().astype(np.float64)
            err = np.abs(fa - fb) / np.maximum(np.abs(fb), 1e-12)
            assert err[~solid].max() <= 1e-5
            assert a.mass_stats()["rescaleCount"] == b.mass_stats()["rescaleCount"] and not a.mass_stats()["hasNaN"]
            assert abs(a.read_forces().fx - b.read_forces().fx) <= 1e-4 * abs(b.read_forces().fx)
    batch.close()
    for es in made:
        for e in es:
            e.close()


@pytest.mark.parametrize("change", ["lattice", "precision"])
def test_another_lattice_or_precision_is_refused(gpu_engine_cls, change):
    es = [gpu_engine_cls(0) for _ in EVEN]
    for e, d in zip(es, EVEN):
        _voxelize(e, d, 0.5)
    batch = LBMBatch(es)
    batch.step(3)
    if change == "lattice":
        _voxelize(es[1], (128, 32, 24), 0.5)
    else:
        es[1].update_config({"precision": "f16s"})
    for call in (lambda: batch.step(1), lambda: batch.autotune(2)):
        with pytest.raises(AerosimError) as err:
            call()
        assert err.value.code == N.ERR_STATE
    es[1].step(3)  # alone it goes on
    assert not es[1].mass_stats()["hasNaN"]
    batch.close()
    for e in es:
        e.close()
