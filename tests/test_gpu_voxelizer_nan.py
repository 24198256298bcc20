"""Meshes with NaN coordinates, as damaged STL files hold them: the scanlines' hits then hold
NaNs, and what they fill depends on the order in which an insertion sort leaves them, that is
on the order of the traversal and of the triangles in the leaves (bvh.ts:141-253, 375-457,
voxelizer.ts:127-173).  The solid cells are compared with a restatement of both in Python
(double precision, the same operations), and one call with the next."""
import math

import numpy as np
import pytest

from aerosim_b200 import meshes

NAN = math.nan
GRID, HEIGHT = (48, 24, 26), 2.4


def _tree(tri):
    """Triangle order and nodes (box, first or children, count) of the reference's build."""
    cen = [[(a[k] + b[k] + c[k]) / 3.0 for k in range(3)] for a, b, c in tri]
    lo = [[NAN if any(math.isnan(v[k]) for v in t) else min(v[k] for v in t) for k in range(3)] for t in tri]
    hi = [[NAN if any(math.isnan(v[k]) for v in t) else max(v[k] for v in t) for k in range(3)] for t in tri]
    order, nodes = list(range(len(tri))), [None]

    def build(n, first, count):
        box, cb = [[math.inf] * 3, [-math.inf] * 3], [[math.inf] * 3, [-math.inf] * 3]
        for t in order[first:first + count]:
            for k in range(3):
                if lo[t][k] < box[0][k]: box[0][k] = lo[t][k]
                if hi[t][k] > box[1][k]: box[1][k] = hi[t][k]
                if cen[t][k] < cb[0][k]: cb[0][k] = cen[t][k]
                if cen[t][k] > cb[1][k]: cb[1][k] = cen[t][k]
        nodes[n] = (box, first, count)
        ext = [cb[1][k] - cb[0][k] for k in range(3)]
        axis = 0
        for k in (1, 2):
            if ext[k] > ext[axis]: axis = k
        if count <= 4 or ext[axis] <= 1e-12:
            return
        split, i, j = 0.5 * (cb[0][axis] + cb[1][axis]), first, first + count - 1
        while i <= j:
            if cen[order[i]][axis] < split:
                i += 1
            else:
                order[i], order[j] = order[j], order[i]
                j -= 1
        left = i - first
        if left in (0, count): left = count >> 1
        child = len(nodes)
        nodes.extend([None, None])
        nodes[n] = (box, child, 0)
        build(child, first, left)
        build(child + 1, first + left, count - left)

    build(0, 0, len(tri))
    return order, nodes


def _hits(tri, order, nodes, y, z):
    py, pz, hits, stack = y + 1.37e-8, z + 2.93e-8, [], [0]
    while stack:
        box, first, count = nodes[stack.pop()]
        if py < box[0][1] or py > box[1][1] or pz < box[0][2] or pz > box[1][2]:
            continue
        if count == 0:
            stack += [first + 1, first]
            continue
        for t in order[first:first + count]:
            a, b, c = tri[t]
            e1, e2 = [b[k] - a[k] for k in range(3)], [c[k] - a[k] for k in range(3)]
            det = -e1[1] * e2[2] + e1[2] * e2[1]
            if abs(det) < 1e-13:
                continue
            inv, ty, tz = 1.0 / det, py - a[1], pz - a[2]
            u = (-ty * e2[2] + tz * e2[1]) * inv
            if u < 0.0 or u > 1.0:
                continue
            v = (ty * e1[2] - tz * e1[1]) * inv
            if v < 0.0 or u + v > 1.0:
                continue
            hits.append(a[0] + u * e1[0] + v * e2[0])
    for i in range(1, len(hits)):
        key, j = hits[i], i - 1
        while j >= 0 and hits[j] > key:
            hits[j + 1] = hits[j]
            j -= 1
        hits[j + 1] = key
    return hits


def _solid_rows(pos):
    """(iy, iz) -> solid cells of the row; rows whose odd count has finite ends are left out
    (they go to the three-ray vote).  Also the number of rows with a NaN among their hits."""
    nx, ny, nz = GRID
    tri = [[[float(x) for x in v] for v in t] for t in pos.reshape(-1, 3, 3)]
    order, nodes = _tree(tri)
    h = HEIGHT / ny
    o = [-n * h * 0.5 for n in GRID]
    box = nodes[0][0]
    w0 = [max(0, math.floor((box[0][k] - o[k]) / h) - 1) for k in range(3)]
    w1 = [min(n - 1, math.ceil((box[1][k] - o[k]) / h) + 1) for k, n in enumerate(GRID)]
    rows, with_nan = {}, 0
    for iz in range(nz):
        for iy in range(ny):
            row = np.zeros(nx, bool)
            if w0[1] <= iy <= w1[1] and w0[2] <= iz <= w1[2]:
                hits = _hits(tri, order, nodes, o[1] + (iy + 0.5) * h, o[2] + (iz + 0.5) * h)
                nan = any(math.isnan(x) for x in hits)
                if len(hits) % 2 and not (math.isnan(hits[0]) or math.isnan(hits[-1])):
                    continue
                with_nan += nan
                if len(hits) % 2 == 0:
                    for a, b in zip(hits[::2], hits[1::2]):
                        if b - a < 1e-7 or math.isnan(a) or math.isnan(b):
                            continue
                        s, e = max(w0[0], math.ceil((a - o[0]) / h - 0.5)), min(w1[0], math.floor((b - o[0]) / h - 0.5))
                        row[s:max(s, e + 1)] = True
            rows[iy, iz] = row
    return rows, with_nan


def _plate(x):
    return [(x, -0.9, -0.9), (x, 0.9, -0.9), (x, 0.0, 0.9)]


def _box():
    pos, idx = meshes.box(1.0, 0.8, 0.9, 4)
    return np.asarray(pos, np.float32)[np.asarray(idx).ravel()] if idx is not None else np.asarray(pos, np.float32)


def _mesh(name):
    if name.startswith("plates"):
        return np.array(sum((_plate({"n": NAN, "a": -0.5, "b": 0.5, "c": 0.8}[c]) for c in name[7:]), []), np.float32)
    box = _box()
    plate = np.array(_plate(NAN), np.float32)
    if name == "box and plates":  # two in different places of the list
        return np.concatenate([box[:150], plate, box[150:], plate])
    if name == "box and plates first":
        return np.concatenate([plate, plate, plate, plate, box])
    r = np.random.default_rng(3)
    box[r.integers(0, len(box), 9), 1 if name == "box without some y" else 0] = NAN
    return box


NAMES = ["plates nnab", "plates anbn", "plates nab", "plates abn", "plates nanbnc", "plates cnbnan", "box and plates",
         "box and plates first", "box without some x", "box without some y"]


def test_restatement_on_a_plain_box(oracle_mod):
    pos = _box()
    rows, with_nan = _solid_rows(pos)
    v = oracle_mod.voxelize((pos, None), None, HEIGHT, *GRID)
    got = (v.flags == 1).reshape(GRID[2], GRID[1], GRID[0])
    assert with_nan == 0 and got.sum() > 500
    for (iy, iz), row in rows.items():
        assert np.array_equal(got[iz, iy], row)


@pytest.mark.gpu
@pytest.mark.parametrize("name", NAMES)
def test_solid_cells_of_a_mesh_with_nan(gpu_engine_cls, name):
    pos = _mesh(name)
    rows, with_nan = _solid_rows(pos)
    assert with_nan > 10
    tunnel = {"length": GRID[0] * HEIGHT / GRID[1], "width": GRID[2] * HEIGHT / GRID[1], "height": HEIGHT}
    first = None
    for _ in range(3):
        e = gpu_engine_cls(0)
        e.voxelize((pos, None), None, tunnel, dict(zip(("nx", "ny", "nz"), GRID)))
        g = e.read_voxel_grid()
        e.close()
        got = (g.cellFlags == 1).reshape(GRID[2], GRID[1], GRID[0])
        for (iy, iz), row in rows.items():
            assert np.array_equal(got[iz, iy], row), (iy, iz)
        assert g.solidCellCount == got.sum()
        if first is None:
            first = g
        assert np.array_equal(g.cellFlags, first.cellFlags) and np.array_equal(g.boundaryQValues, first.boundaryQValues)
