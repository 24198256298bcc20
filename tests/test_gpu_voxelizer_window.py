"""The voxelizer's window where the mesh's bounds leave the int range of cell indices: a mesh
beside the lattice gives an empty grid however far it reaches along another axis."""
import numpy as np
import pytest

from test_gpu_voxelizer import _compare

pytestmark = pytest.mark.gpu

GRID, H = (48, 24, 26), 2.4


@pytest.mark.parametrize("axis,beside,sign", [(0, 1, 1), (0, 2, -1), (1, 0, 1), (2, 1, -1)])
def test_far_reaching_mesh_beside_the_lattice(gpu_engine_cls, oracle_mod, axis, beside, sign):
    nx, ny, nz = GRID
    tri = np.zeros((3, 3), np.float32)
    tri[:, axis] = (0.1, 1e30, 0.1)   # its window starts inside the lattice and wraps
    tri[:, beside] = sign * np.array([5.0, 5.5, 6.0], np.float32)
    tri[2, 3 - axis - beside] = 0.5
    e = gpu_engine_cls(0)
    e.voxelize((tri, None), None, {"length": 4.8, "width": 2.6, "height": H}, {"nx": nx, "ny": ny, "nz": nz})
    g = e.read_voxel_grid()
    assert g.solidCellCount == 0 and g.boundaryCellCount == 0 and not g.cellFlags.any()
    _compare(g, oracle_mod.voxelize((tri, None), None, H, nx, ny, nz))
    e.close()
