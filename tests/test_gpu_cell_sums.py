"""Cell sums of FP32 positions: a batch sums centroids and perimeters in fixed point where that is exact,
a small sphere in FP64 (one and two threads a cell), and both give the same bits -- also where the
fixed-point sum gives way: coordinates that are zero, subnormal or far below the radius, and edges of
no length."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [57, 120, 333, 1200]
SEEDS = [3, 4, 5, 6]


@pytest.mark.parametrize("tiny", [None, 0.0, -0.0, 1e-42, -1e-30, 1e-12, 3e-8, 1e-6])
def test_fixed_point_and_fp64_sums_agree_bitwise(svm_lib, tiny):
    svm = svm_lib
    if svm.device_count() < 1:
        pytest.fail("no CUDA device: the GPU tests need a GB300")
    b = svm.sphericalVertexModelBatch(SIZES, SEEDS, p0=3.8)
    pos = b.returnPositions()
    rng = np.random.default_rng(2)
    for r in range(len(SIZES)):
        p = pos[b.vertexSlice(r)]
        p[:] *= 1.0 + 1e-3 * rng.standard_normal(p.shape)
        if tiny is not None:            # the coordinates nearest to zero, in each direction
            for d in range(3):
                p[np.argsort(np.abs(p[:, d]))[:9], d] = tiny
            n = b.vertexNeighbors()[b.vertexSlice(r)][0, 0] - b.vertexSlice(r).start
            p[n] = p[0]                 # an edge of length zero
    b.setPositions(pos)
    b.computeGeometry()
    cells, ap = b.cellPositions(), b.areaPerimeter()
    for r in range(len(SIZES)):
        noise = svm.noiseSource()
        noise.setReproducibleSeed(SEEDS[r])
        m = svm.sphericalVertexModel(SIZES[r], noise, 1.0, 3.8)
        m.precision = "mixed"
        m.setPositions(pos[b.vertexSlice(r)])
        m.computeGeometry()
        assert np.array_equal(cells[b.cellSlice(r)], m.cellPositions())
        a, e = ap[b.cellSlice(r)], m.areaPerimeter()
        assert np.array_equal(a[:, 1], e[:, 1])
        # (an area check that fails replaces areas by the fan's, for both; NaN areas compare as such)
        assert np.array_equal(a[:, 0], e[:, 0], equal_nan=True)
