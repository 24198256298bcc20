"""The two-cell step's plain chunks: 32 pairs without a solid, near-wall or wall-row cell, in a
step that writes no macro field.  They have a code path of their own (unconditional pair
stores that the row ends overwrite, a density sum without per-cell tests), which a call's last
step never takes, as it writes the macro fields.

So n steps in one call, n - 1 of them with plain chunks, are compared with n calls of one step,
which have none: both store the same collision's values, add the same fixed-point densities and
so take the same rescale decisions, and every bit agrees.  (One step of the other path is
compared with the one-cell kernel in test_gpu_pair_items.py.)  The mean density starts 0.3 %
high, so that each step's sum decides on a rescale that the next step applies."""
import numpy as np
import pytest

from aerosim_b200 import LBMBatch, VoxelGridResult, sgs
from test_gpu_pair_items import C, W

PRECISIONS = ["f32", "f16s", "f16c", "bf16s"]
SMS = 148


def _flags(nx, ny, nz):
    """A block of 2 x 2 x 1 solids in the middle and the cells around it."""
    solid = np.zeros((nz, ny, nx), bool)
    solid[nz // 2, ny // 2:ny // 2 + 2, nx // 2 - 1:nx // 2 + 1] = True
    near = np.zeros_like(solid)
    for c in C[1:]:
        near |= np.roll(solid, tuple(-c[::-1]), (0, 1, 2))
    return np.where(solid, 1, np.where(near, 2, 0)).astype(np.uint8)


def _item_rows(nx, rows, pairs):
    r = min(pairs // (nx // 2), -(-rows // (2 * SMS)))
    return max(1, min(16, r))


def _plain_chunks(flags, r):
    """(row ends in plain chunks, of these in a ragged last item) for items of r rows."""
    nz, ny, nx = flags.shape
    np_, rows = nx // 2, ny * nz
    f = flags.reshape(rows, nx)[:, :2 * np_] != 0
    iy, iz = np.arange(rows) % ny, np.arange(rows) // ny
    f[(iy == 0) | (iy == ny - 1) | ((nz > 4) & ((iz == 0) | (iz == nz - 1)))] = True
    pair = f.reshape(rows, np_, 2).any(2)
    ends = ragged = 0
    for r0 in range(0, rows, r):
        item = pair[r0:r0 + r].ravel()
        for c in range(0, len(item), 32):
            if not item[c:c + 32].any():
                x = np.arange(c, min(c + 32, len(item))) % np_
                n = int((x == 0).sum() + (x == np_ - 1).sum())
                ends += n
                if r0 + r > rows:
                    ragged += n
    return ends, ragged


def _populations(nx, ny, nz, seed=5):
    g, n = np.random.default_rng(seed), nx * ny * nz
    u = 0.03 * g.standard_normal((3, n)) + np.array([[0.06], [0], [0]])
    cu = 3 * C @ u
    rho = 1.003 + 0.002 * g.standard_normal(n)
    f = W[:, None] * rho * (1 + cu + 0.5 * cu * cu - 1.5 * (u * u).sum(0)) + 1e-4 * W[:, None] * g.standard_normal((19, n))
    return f.astype(np.float32)


def _engine(cls, dims, precision, closure=False):
    nx, ny, nz = dims
    flags = _flags(nx, ny, nz).ravel()
    cells = np.flatnonzero(flags == 2).astype(np.int32)
    q = np.random.default_rng(1).uniform(0.01, 1.0, (len(cells), 18)).astype(np.float32)
    bmap = np.full(flags.size, -1, np.int32)
    bmap[cells] = np.arange(len(cells))
    e = cls(0)
    e.set_voxel_grid(VoxelGridResult(nx, ny, nz, 1.0, 1.0, 1.0, -nx / 2, -ny / 2, -nz / 2, flags, bmap, cells, q.ravel(),
                                     q.min(1), int((flags == 1).sum()), len(cells), 0, 0.0),
                     {"uInletLattice": 0.06, "nuLattice": 0.0005, "smagorinskyCs": 0.1, "precision": precision,
                      "tunnel": {"length": nx, "width": nz, "height": ny}})
    if closure:
        e.set_sgs_mlp(sgs.init_params(3))
    return e


def _same(a, b):
    assert np.array_equal(a.read_populations().view(np.uint32), b.read_populations().view(np.uint32))
    ma, mb = a.mass_stats(), b.mass_stats()
    assert repr(ma) == repr(mb)  # NaN sums included
    return ma


LATTICES = [(32, 893, 4), (66, 301, 4), (130, 100, 12), (4, 1003, 4), (6, 1003, 4), (258, 40, 12)]
ODD = [(33, 893, 4), (65, 301, 4), (129, 100, 12), (5, 1003, 4), (7, 1003, 4), (257, 40, 12)]


def _pairs(precision, closure):
    return 384 if precision != "f32" else 256 if closure else 192


def test_lattices_have_the_chunks():
    for dims in LATTICES + ODD:
        flags = _flags(*dims)
        for pairs in (192, 256, 384):
            assert _plain_chunks(flags, _item_rows(dims[0], dims[1] * dims[2], pairs))[0] > 100, dims
    for pairs in (192, 256, 384):  # and for each item size some in a ragged last item, even and odd
        for group in (LATTICES, ODD):
            assert any(_plain_chunks(_flags(*d), _item_rows(d[0], d[1] * d[2], pairs))[1] for d in group)


@pytest.mark.gpu
@pytest.mark.parametrize("closure", [False, True], ids=["", "closure"])
@pytest.mark.parametrize("precision", PRECISIONS)
@pytest.mark.parametrize("dims", LATTICES + ODD, ids=lambda d: f"{d[0]}x{d[1]}x{d[2]}")
def test_plain_chunks_of_a_lattice(gpu_engine_cls, dims, precision, closure):
    f = _populations(*dims)
    one, many = (_engine(gpu_engine_cls, dims, precision, closure) for _ in range(2))
    for e in (one, many):
        e.write_populations(f)
    for n in (2, 3):  # non-macro steps of both parities
        one.step(n)
        for _ in range(n):
            many.step(1)
        stats = _same(one, many)
    assert stats["rescaleCount"] > 0 and not stats["hasNaN"]
    one.close(), many.close()


@pytest.mark.gpu
@pytest.mark.parametrize("precision", PRECISIONS)
@pytest.mark.parametrize("dims,cell", [((66, 301, 4), (0, 40, 1)), ((66, 301, 4), (64, 40, 1)), ((65, 301, 4), (64, 40, 1)),
                                       ((130, 100, 12), (77, 50, 3))], ids=str)
def test_nan_in_a_plain_chunk(gpu_engine_cls, dims, precision, cell):
    """A NaN density adds nothing to the sum and is reported, on either path; the row ends' too."""
    nx, ny, nz = dims
    f = _populations(*dims)
    f[:, cell[0] + nx * (cell[1] + ny * cell[2])] = np.nan
    one, many = (_engine(gpu_engine_cls, dims, precision) for _ in range(2))
    for e in (one, many):
        e.write_populations(f)
    one.step(3)
    for _ in range(3):
        many.step(1)
    a, b = one.read_populations(), many.read_populations()
    assert np.isnan(a).any()
    assert np.array_equal(a, b, equal_nan=True)
    sa, sb = one.mass_stats(), many.mass_stats()
    assert sa["hasNaN"] and sb["hasNaN"]
    assert sa["rescaleCount"] == sb["rescaleCount"] and sa["cumulativeRescale"] == sb["cumulativeRescale"]
    one.close(), many.close()


BATCHES = {"one pitch": [(66, 301, 4), (80, 120, 8)], "pitches": [(32, 500, 4), (130, 100, 12), (6, 403, 4), (258, 40, 12)],
           "odd and even": [(65, 301, 4), (66, 201, 4), (129, 60, 9)]}


@pytest.mark.gpu
@pytest.mark.parametrize("item_cells", [256, 1024])
@pytest.mark.parametrize("precision", PRECISIONS)
@pytest.mark.parametrize("name", list(BATCHES))
def test_plain_chunks_of_a_batch(gpu_engine_cls, name, precision, item_cells):
    made = []
    for calls in ((2, 3), (1,) * 5):
        es = [_engine(gpu_engine_cls, d, precision) for d in BATCHES[name]]
        b = LBMBatch(es)
        b.set_tuning(2, 1, 1, item_cells)
        for k, (e, d) in enumerate(zip(es, BATCHES[name])):
            e.write_populations(_populations(*d, seed=5 + k))
        for n in calls:
            b.step(n)
        made.append((b, es))
    for one, many in zip(made[0][1], made[1][1]):
        stats = _same(one, many)
        assert stats["rescaleCount"] > 0 and not stats["hasNaN"]
    for b, es in made:
        b.close()
        for e in es:
            e.close()
