"""The device-built tree and the arrays an engine keeps between voxelizations: grids bit for
bit against the oracle at the sizes where the build changes its way (leaves of 4, subtrees
of 128 triangles, CTAs of 512 threads), on lopsided and coincident triangles and where it
hands back to the host build, and on one engine after another body, lattice and failure."""
import numpy as np
import pytest

from aerosim_b200 import AerosimError, meshes, voxelize_mesh_to_lattice
from test_gpu_voxelizer import _compare

pytestmark = pytest.mark.gpu

GRID = (48, 24, 26)


def _check(oracle_mod, mesh, world=None, height=2.4, dims=GRID):
    nx, ny, nz = dims
    tunnel = {"length": nx * height / ny, "width": nz * height / ny, "height": height}
    gpu = voxelize_mesh_to_lattice(mesh, world, tunnel, {"nx": nx, "ny": ny, "nz": nz})
    _compare(gpu, oracle_mod.voxelize(mesh, world, height, nx, ny, nz))
    return gpu


def _soup(n, seed, size=0.5):
    """n random triangles: any number of hits per scanline, so votes and fills mix."""
    r = np.random.default_rng(seed)
    c = r.uniform(-0.9, 0.9, (n, 1, 3))
    return ((c + r.uniform(-size, size, (n, 3, 3))).reshape(-1, 3).astype(np.float32), None)


@pytest.mark.parametrize("n", [1, 4, 5, 127, 128, 129, 511, 513, 1500])
def test_triangle_counts(gpu_engine_cls, oracle_mod, n):
    _check(oracle_mod, _soup(n, n, 0.5 if n < 200 else 0.08))


def test_closed_body_of_many_triangles(gpu_engine_cls, oracle_mod):
    g = _check(oracle_mod, meshes.uv_sphere(0.8, 160, 120), dims=(60, 31, 33))
    assert g.solidCellCount > 1000


@pytest.mark.parametrize("copies", [3, 40, 50])
def test_coincident_triangles(gpu_engine_cls, oracle_mod, copies):
    """Equal centroids end in one leaf whatever their number (a box repeated `copies` times:
    at most 2 x 50 hits a scanline)."""
    pos, idx = meshes.box(1.0, 0.8, 0.9, 1)
    _check(oracle_mod, (pos, np.tile(idx, (copies, 1))))


def test_lopsided_tree(gpu_engine_cls, oracle_mod):
    """Plates at x = 2^-k: every split takes one off."""
    p = []
    for k in range(30):
        x = 0.9 * 2.0 ** -k
        p += [(x, -0.9, -0.9), (x, 0.9, -0.9), (x, 0.0, 0.9)]
    _check(oracle_mod, (np.array(p, np.float32), None))


def test_split_that_leaves_one_side_empty(gpu_engine_cls, oracle_mod):
    """Centroids one rounding apart far from the origin: the split falls on the lower one."""
    m = np.diag([1e-10, 1e-13, 1e-13, 1.0])
    m[0, 3] = 1e6
    _check(oracle_mod, _soup(200, 5), m.T.reshape(-1).copy(), height=4e6)


def test_too_deep_a_tree_is_refused_and_the_engine_goes_on(gpu_engine_cls, oracle_mod):
    h = 3.0 ** 48
    p, e = [], 0.25 * h
    for k in range(-24, 48):  # one plate off per split: 68 left turns, more siblings wait than the stack holds
        x = 3.0 ** k
        p += [(x, -e, -e), (x, e, -e), (x, 0.0, e)]
    nx, ny, nz = GRID
    tunnel, grid = {"length": 2 * h, "width": h, "height": h}, {"nx": nx, "ny": ny, "nz": nz}
    box = meshes.box(0.4 * h, 0.3 * h, 0.3 * h, 2)
    eng = gpu_engine_cls(0)
    eng.voxelize(box, None, tunnel, grid)
    with pytest.raises(AerosimError) as err:
        eng.voxelize((np.array(p, np.float32), None), None, tunnel, grid)
    assert err.value.code == -4 and "stack" in str(err.value)
    _compare(eng.read_voxel_grid(), oracle_mod.voxelize(box, None, h, nx, ny, nz))
    eng.close()


def test_bounds_beyond_the_index_range_are_refused(gpu_engine_cls, oracle_mod):
    """A triangle 1e30 long: the window's cell counts leave the int range."""
    nx, ny, nz = GRID
    tunnel, grid = {"length": 4.8, "width": 2.6, "height": 2.4}, {"nx": nx, "ny": ny, "nz": nz}
    box = meshes.box(1.0, 0.8, 0.9, 2)
    eng = gpu_engine_cls(0)
    eng.voxelize(box, None, tunnel, grid)
    far = np.array([(0.1, 0.0, 0.0), (1e30, 0.5, 0.0), (0.1, 0.0, 0.5)], np.float32)
    with pytest.raises(AerosimError) as err:
        eng.voxelize((far, None), None, tunnel, grid)
    assert err.value.code == -3 and "bounds" in str(err.value)
    _compare(eng.read_voxel_grid(), oracle_mod.voxelize(box, None, 2.4, nx, ny, nz))
    eng.close()


def test_engine_reused_for_other_bodies_and_lattices(gpu_engine_cls, oracle_mod):
    """One engine through several bodies and lattices steps like fresh ones, with the flow
    reset or kept."""
    bodies = [(meshes.box(1.0, 0.8, 0.9, 2), (48, 24, 26)), (meshes.uv_sphere(0.6, 40, 30), (48, 24, 26)),
              (meshes.box(0.4, 0.5, 0.3, 2), (48, 24, 26)), (meshes.uv_sphere(0.5, 40, 30), (65, 24, 31)),
              (meshes.box(1.0, 0.8, 0.9, 2), (48, 24, 26))]
    cfg = {"uInletLattice": 0.06, "nuLattice": 0.004, "smagorinskyCs": 0.1, "precision": "f32"}

    def start(e, body, dims, reset=True):
        tunnel = {"length": dims[0] * 0.1, "width": dims[2] * 0.1, "height": dims[1] * 0.1}
        e.voxelize(body, None, tunnel, dict(zip(("nx", "ny", "nz"), dims)), cfg, reset_flow=reset)
        return e

    one = gpu_engine_cls(0)
    for body, dims in bodies:
        start(one, body, dims).step(7)
        fresh = start(gpu_engine_cls(0), body, dims)
        fresh.step(7)
        a, b = one.read_populations(), fresh.read_populations()
        assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
        _compare(one.read_voxel_grid(), oracle_mod.voxelize(body, None, dims[1] * 0.1, *dims))
        fresh.close()
    # the body changes under a running flow: populations stay
    kept = one.read_populations()
    start(one, bodies[1][0], bodies[1][1], reset=False)
    assert np.array_equal(one.read_populations().view(np.uint32), kept.view(np.uint32))
    one.step(3)
    assert not one.mass_stats()["hasNaN"]
    one.close()
