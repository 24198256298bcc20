"""The two-cells-per-thread step at the edges of its work items: rows shorter and longer than
a warp's 32 pairs, items that cross iz planes (also several of them), up to 16 rows an item, a
ragged last item, solid and near-wall cells at the row ends and in every chunk, macro steps,
batches of one and of several row pitches, rows of an odd cell count, the learned closure.

Each lattice holds random solids and random populations; one step of it is compared with the
one-cell-per-thread kernel's.  The two round differently: about 60 FP32 operations on values
below 1/3 end less than 1e-6 apart; 16-bit storage may then round to the neighbouring value,
one storage ulp of the largest deviation, and F16C adds the 18 directions' rounding errors to
direction 0.
"""
import numpy as np
import pytest

from aerosim_b200 import LBMBatch, LBMEngine, VoxelGridResult, sgs

pytestmark = pytest.mark.gpu

C = np.array([(0, 0, 0), (1, 0, 0), (-1, 0, 0), (0, 1, 0), (0, -1, 0), (0, 0, 1), (0, 0, -1), (1, 1, 0), (-1, -1, 0),
              (1, -1, 0), (-1, 1, 0), (1, 0, 1), (-1, 0, -1), (1, 0, -1), (-1, 0, 1), (0, 1, 1), (0, -1, -1),
              (0, 1, -1), (0, -1, 1)])
W = np.array([1 / 3] + [1 / 18] * 6 + [1 / 36] * 12)
ULPS = {"f32": 0.0, "f16s": 2.0**-10, "f16c": 19 * 2.0**-10, "bf16s": 2.0**-7}


def _lattice(nx, ny, nz, precision, ground):
    g = np.random.default_rng(nx + 1000 * ny)
    n = nx * ny * nz
    solid = g.random((nz, ny, nx)) < 0.05
    near = np.zeros_like(solid)
    for c in C[1:]:
        near |= np.roll(solid, tuple(-c[::-1]), (0, 1, 2))
    flags = np.where(solid, 1, np.where(near, 2, 0)).astype(np.uint8).ravel()
    cells = np.flatnonzero(flags == 2).astype(np.int32)
    q = g.uniform(0.01, 1.0, (len(cells), 18)).astype(np.float32)
    bmap = np.full(n, -1, np.int32)
    bmap[cells] = np.arange(len(cells))
    e = LBMEngine(0)
    e.set_voxel_grid(VoxelGridResult(nx, ny, nz, 1.0, 1.0, 1.0, -nx / 2, -ny / 2, -nz / 2, flags, bmap, cells, q.ravel(),
                                     q.min(1), int(solid.sum()), len(cells), 0, 0.0),
                     {"uInletLattice": 0.06, "nuLattice": 0.0005, "smagorinskyCs": 0.1, "precision": precision,
                      "groundNoSlip": ground, "tunnel": {"length": nx, "width": nz, "height": ny}})
    u = 0.04 * g.standard_normal((3, n)) + np.array([[0.06], [0], [0]])
    cu = 3 * C @ u
    rho = 1 + 0.002 * g.standard_normal(n)
    f = W[:, None] * rho * (1 + cu + 0.5 * cu * cu - 1.5 * (u * u).sum(0)) + 1e-4 * W[:, None] * g.standard_normal((19, n))
    e.write_populations(f.astype(np.float32))
    return e, flags


def _compare(two, one, flags, precision, tol=1e-6):
    a = two.read_populations().reshape(19, -1).astype(np.float64)
    b = one.read_populations().reshape(19, -1).astype(np.float64)
    tol += ULPS[precision] * np.abs(b - W[:, None])[:, flags != 1].max()
    assert np.abs(a - b)[:, flags != 1].max() <= tol
    ma, mb = two.read_macro(), one.read_macro()
    for k in ("ux", "uy", "uz", "rho"):  # read from the same source lattice by both
        assert np.abs(ma[k] - mb[k]).max() <= 2e-6, k
    sa, sb = two.mass_stats(), one.mass_stats()
    assert abs(sa["meanRho"] - sb["meanRho"]) <= 1e-7 and sa["rescaleCount"] == sb["rescaleCount"]


LATTICES = [(4, 7, 3, False), (6, 5, 950, True), (30, 40, 44, False), (34, 7, 200, True), (62, 9, 66, False),
            (66, 31, 21, True), (130, 12, 400, False), (10, 3, 1600, False), (386, 6, 5, True)]


@pytest.mark.parametrize("precision", list(ULPS))
@pytest.mark.parametrize("dims", LATTICES, ids=lambda d: f"{d[0]}x{d[1]}x{d[2]}")
def test_items_of_a_lattice(gpu_engine_cls, monkeypatch, dims, precision):
    e = {}
    for cpt in (1, 2):
        monkeypatch.setenv("AEROSIM_CELLS_PER_THREAD", str(cpt))
        e[cpt], flags = _lattice(*dims[:3], precision, dims[3])
        e[cpt].step(1)
    _compare(e[2], e[1], flags, precision)
    for x in e.values():
        x.close()


ODD = [(5, 9, 8, False), (7, 9, 300, True), (63, 44, 31, False), (65, 7, 200, True), (129, 12, 400, False),
       (385, 6, 5, True)]


@pytest.mark.parametrize("precision", list(ULPS))
@pytest.mark.parametrize("dims", ODD, ids=lambda d: f"{d[0]}x{d[1]}x{d[2]}")
def test_rows_of_an_odd_cell_count_keep_their_bits(gpu_engine_cls, monkeypatch, dims, precision):
    e = {}
    for cpt in (1, 2):
        monkeypatch.setenv("AEROSIM_CELLS_PER_THREAD", str(cpt))
        e[cpt], flags = _lattice(*dims[:3], precision, dims[3])
        e[cpt].step(1)
    _compare(e[2], e[1], flags, precision)
    for x in e.values():
        x.step(2)
    if precision != "f32":
        assert np.array_equal(e[1].read_populations(), e[2].read_populations())
    for x in e.values():
        x.close()


@pytest.mark.parametrize("precision", list(ULPS))
@pytest.mark.parametrize("dims", [(4, 7, 3, False), (62, 9, 66, True), (66, 31, 21, False), (130, 12, 100, False),
                                  (256, 6, 7, True), (5, 9, 8, False), (65, 7, 100, True)],
                         ids=lambda d: f"{d[0]}x{d[1]}x{d[2]}")
def test_items_with_the_closure(gpu_engine_cls, monkeypatch, dims, precision):
    # an input that rounds to the neighbouring BF16 value (2^-8 of the eddy viscosity) moves a
    # population by less than 4.5/18 |Pi| 2^-8, 1e-6 for the stresses here
    e = {}
    for cpt in (1, 2):
        monkeypatch.setenv("AEROSIM_CELLS_PER_THREAD", str(cpt))
        e[cpt], flags = _lattice(*dims[:3], precision, dims[3])
        f = e[cpt].read_populations()
        e[cpt].set_sgs_mlp(sgs.init_params(3))
        e[cpt].write_populations(f)
        e[cpt].step(1)
    _compare(e[2], e[1], flags, precision, tol=2e-6)
    for x in e.values():
        x.close()


@pytest.mark.parametrize("precision", list(ULPS))
@pytest.mark.parametrize("dims", [[(4, 5, 6), (34, 9, 40), (130, 12, 30)], [(66, 31, 21), (72, 7, 50)]],
                         ids=["pitches", "one_pitch"])
def test_items_of_a_batch(gpu_engine_cls, monkeypatch, dims, precision):
    made = {}
    for cpt in (1, 2):
        monkeypatch.setenv("AEROSIM_CELLS_PER_THREAD", str(cpt))
        made[cpt] = [_lattice(*d, precision, False) for d in dims]
        b = LBMBatch([e for e, _ in made[cpt]])
        b.set_tuning(2, 2, 1, 512)
        b.step(1)
        b.close()
    for (two, flags), (one, _) in zip(made[2], made[1]):
        _compare(two, one, flags, precision)
        two.close(), one.close()
