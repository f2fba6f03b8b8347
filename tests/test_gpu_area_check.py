"""The mixed form's total-area check: rounding alone does not take the triangle-fan fallback, however many
cells it adds up over, and a wrapped angle does at any size."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _sphere(svm, n):
    rng = np.random.default_rng(n)
    i = np.arange(n) + 0.5
    z = 1 - 2 * i / n
    s, phi = np.sqrt(1 - z * z), np.pi * (3 - np.sqrt(5)) * i
    p = np.stack([s * np.cos(phi), s * np.sin(phi), z], 1) + rng.normal(0, 0.1 * np.sqrt(4 * np.pi / n), (n, 3))
    p *= np.sqrt(n / (4 * np.pi)) / np.linalg.norm(p, axis=1, keepdims=True)
    m = svm.sphericalVertexModel(n, topology=svm.Topology(p, device=True))
    m.precision = "mixed"
    return m


@pytest.mark.parametrize("n", [1000, 137000, 400000])
def test_limit(svm_lib, n):
    m = _sphere(svm_lib, n)
    R = m.radius
    m.computeGeometry()
    total, excess, taken = m.areaCheck()
    limit = max(1e-6, 6 * n * R * R * 2.0 ** -53)
    assert taken == (abs(excess) > limit) and not taken
    assert abs(m.areaPerimeter()[:, 0].sum() - 4 * np.pi * R * R) < 1e-3
    # forty vertices carried far past a neighbour: some of the angles wrap, by whole multiples of pi
    # (15 of them at 20,000 cells in the CPU restatement)
    pos, nb = m.returnPositions(), m.vertexNeighbors()
    for v in range(11, 11 + 40 * 37, 37):
        u = nb[v][0]
        q = pos[u] + 4.0 * (pos[u] - pos[v])
        pos[v] = R * q / np.linalg.norm(q)
    m.setPositions(pos)
    m.computeGeometry()
    _, excess, taken = m.areaCheck()
    assert abs(excess) > 0.5 * np.pi * R * R and taken
