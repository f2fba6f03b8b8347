"""Perimeters of FP32 positions whose edges span more bits than a double holds: the sum in fixed point (a batch) gives
way to the FP64 sum of a small sphere, whose roundings are the reference's order."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_perimeters_of_long_cells_with_tiny_edges(svm_lib):
    svm = svm_lib
    if svm.device_count() < 1:
        pytest.fail("no CUDA device: the GPU tests need a GB300")
    seeds = range(3, 67)
    topos = [svm.Topology(svm.random_cell_centres(s, 57 + s % 24)) for s in seeds]
    rng = np.random.default_rng(9)
    pos, long = [], []
    for t in topos:
        p, R = t.vertexPositions.copy(), t.radius
        c = int(np.flatnonzero(t.ringCounts == 5)[0])
        ring = t.rings[c, :5]
        # two edges of 2^-27 to 2^-26 (units of 2^-50), which the sum takes last, and three of a quarter circle (a
        # sum from 10 on: rounded to 2^-49 and more)
        d, a = rng.uniform(7.5e-9, 1.45e-8, 2), rng.uniform(0, 2 * np.pi, 2)
        p[ring[:3]] = [[R, 0, 0], [R, d[0] * np.cos(a[0]), d[0] * np.sin(a[0])],
                       [R, d @ np.cos(a), d @ np.sin(a)]]
        p[ring[3]], p[ring[4]] = [0, 0, R], [0, R, 0]
        pos.append(p.astype(np.float32).astype(np.float64))
        long.append(c)
    b = svm.sphericalVertexModelBatch([t.nCells for t in topos], None, topologies=topos)
    b.setPositions(np.concatenate(pos))
    b.computeGeometry()
    ap, cells = b.areaPerimeter(), b.cellPositions()
    for r, t in enumerate(topos):
        m = svm.sphericalVertexModel(t.nCells, topology=t, radius=float(b.radii[r]))
        m.precision = "mixed"
        m.setPositions(pos[r])
        m.computeGeometry()
        mine, one = ap[b.cellSlice(r)], m.areaPerimeter()
        assert one[long[r], 1] > 10
        assert np.array_equal(mine[:, 1], one[:, 1]), (r, mine[long[r], 1] - one[long[r], 1])
        assert np.array_equal(mine[:, 0], one[:, 0], equal_nan=True)
        assert np.array_equal(cells[b.cellSlice(r)], m.cellPositions())
