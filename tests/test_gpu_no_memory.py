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
