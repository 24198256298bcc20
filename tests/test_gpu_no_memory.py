"""Where device memory runs out: a lattice whose populations find none leaves the engine without
a flow, the calls that need one refuse, and the next grid that fits is taken."""
import numpy as np
import pytest

from aerosim_b200 import AerosimError, meshes
from aerosim_b200 import _native as N

pytestmark = pytest.mark.gpu


def _voxelize(e, dims, precision):
    h = dims[1] * 0.1
    e.voxelize(meshes.uv_sphere(0.6, 20, 16), None, {"length": dims[0] * 0.1, "width": dims[2] * 0.1, "height": h},
               dict(zip(("nx", "ny", "nz"), dims)),
               {"uInletLattice": 0.06, "nuLattice": 0.004, "smagorinskyCs": 0.1, "precision": precision})


def test_no_memory_for_the_populations(gpu_engine_cls):
    import torch
    e = gpu_engine_cls(0)
    _voxelize(e, (64, 24, 26), "f32")
    free, _ = torch.cuda.mem_get_info()
    hog = torch.empty(free - (2 << 30), dtype=torch.uint8, device="cuda")
    try:
        with pytest.raises(AerosimError) as err:  # 8.4 M cells: 42 MB of grid fit, 2.6 GB of populations do not
            _voxelize(e, (512, 128, 128), "f64")
        assert err.value.code == N.ERR_NOMEM
        for call in (lambda: e.step(1), e.reset_flow, e.read_forces, e.read_macro, e.mass_stats):
            with pytest.raises(AerosimError) as err:
                call()
            assert err.value.code == N.ERR_STATE
    finally:
        del hog
        torch.cuda.empty_cache()
    fresh = gpu_engine_cls(0)
    for x in (e, fresh):
        _voxelize(x, (128, 32, 32), "f32")
        x.step(4)
    assert np.array_equal(e.read_populations().view(np.uint32), fresh.read_populations().view(np.uint32))
    assert e.read_forces().fx == fresh.read_forces().fx and e.mass_stats() == fresh.mass_stats()
    e.close(), fresh.close()


def test_what_is_kept_for_the_next_grid_goes_back(gpu_engine_cls):
    """After two voxelizations of 33.5 M cells an engine holds the first one's arrays (201 MB)
    for a third.  An allocation that fails gets them, and a small lattice keeps none of them."""
    import torch
    e = gpu_engine_cls(0)
    for _ in range(2):
        _voxelize(e, (512, 256, 256), "f16s")
    free, _ = torch.cuda.mem_get_info()
    hog = torch.empty(free - (100 << 20), dtype=torch.uint8, device="cuda")
    try:
        assert e.read_macro()["rho"].min() > 0.9  # through 134 MB of staging
    finally:
        del hog
        torch.cuda.empty_cache()
    e.close()

    def used_after(grids):
        e = gpu_engine_cls(0)
        before, _ = torch.cuda.mem_get_info()
        for dims in grids:
            _voxelize(e, dims, "f16s")
        after, _ = torch.cuda.mem_get_info()
        e.close()
        return before - after

    used_after([(64, 24, 26)])
    # both keep at most 64 MB of scratch, and the arrays of two grids of 40 000 cells
    assert abs(used_after([(512, 256, 256)] * 3 + [(64, 24, 26)] * 2) - used_after([(64, 24, 26)] * 2)) <= 70 << 20
