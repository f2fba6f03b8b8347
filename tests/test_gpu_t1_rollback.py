"""T1 passes whose parallel flips are undone and replayed in order: sheets with so many short edges that a
flip shortens an edge next to one that has already run.  In one block, over a cluster (the default of spheres
below 50,000 vertices), over a cooperative grid and in a batch, the flips and the connectivity are the CPU
restatement's, and the corners that the pass rebuilds are those of a full evaluation."""
import numpy as np
import pytest

from gpu_helpers import rel_err, same_rings

pytestmark = pytest.mark.gpu

# FP32 positions: each flip that moves a vertex rounds it, to 2^-24 of the radius; 16 roundings of one vertex
TOL = {"fp64": 1e-14, "mixed": 16 * 2.0 ** -24}
CASES = [(2000, 17, 600, 0.04), (400, 6, 300, 0.2), (1000, 8, 900, 0.1)]


def crowded(svm, n, seed, edges):
    """The seeded sphere with `edges` of its edges drawn together to a few per cent."""
    topo = svm.Topology(svm.random_cell_centres(seed, n))
    R = np.sqrt(n / (4 * np.pi))
    rng = np.random.default_rng(seed)
    pos = topo.vertexPositions.copy()
    for v in rng.choice(topo.nVertices, edges, replace=False):
        u = int(topo.vertexNeighbors[v][rng.integers(3)])
        pos[u] = pos[v] + rng.uniform(0.01, 0.05) * (pos[u] - pos[v])
        pos[u] *= R / np.linalg.norm(pos[u])
    return topo, pos, R


def oracle_pass(oracle_mod, topo, pos, R, threshold):
    om = oracle_mod.OracleModel(pos, topo.rings, topo.ringCounts, topo.vertexCells, topo.vertexNeighbors, R)
    om.set_t1_threshold(threshold)
    om.lib.orc_enforce_topology(om.h)
    return om, om.flips()


@pytest.mark.parametrize("form", ["fp64", "mixed"])
@pytest.mark.parametrize("blocks", [0, 1, 4, 64])
@pytest.mark.parametrize("case", CASES)
def test_replayed_pass_matches_oracle(svm_lib, oracle_mod, case, blocks, form):
    svm = svm_lib
    if svm.device_count() < 1:
        pytest.fail("no CUDA device: the GPU tests need a GB300")
    n, seed, edges, threshold = case
    topo, pos, R = crowded(svm, n, seed, edges)
    if form == "mixed":
        pos = pos.astype(np.float32).astype(np.float64)
    m = svm.sphericalVertexModel(n, topology=topo, radius=R)
    m.precision = form
    m.setT1Threshold(threshold)
    m.setT1Blocks(blocks)
    m.setPositions(pos)
    m.enforceTopology()
    om, flips = oracle_pass(oracle_mod, topo, pos, R, threshold)
    stats = m.t1Stats()
    assert stats["rollbacks"] == 1 and stats["flips"] == len(flips) > 100, stats
    assert np.array_equal(m.takeFlips(), flips)
    assert same_rings(m, om, 32)
    assert np.array_equal(m.vertexCellNeighbors(), om.vertex_cells())
    assert np.array_equal(m.vertexNeighbors(), om.vertex_neighbors())
    assert rel_err(m.returnPositions(), om.positions(), R) < TOL[form]
    # a step's pass, whose touched cells' corners the pass rebuilds
    m.loadState(dict(pos=pos, rings=topo.rings, counts=topo.ringCounts, vcells=topo.vertexCells, vnbrs=topo.vertexNeighbors))
    bd = svm.brownianDynamics()
    bd.setModel(m)
    bd.setT(0.0)
    bd.setDeltaT(1e-12)
    bd.integrateEquationOfMotion()
    assert m.t1Stats()["rollbacks"] == 1
    m.computeGeometry()
    patched, p = m.areaPerimeter(), m.returnPositions()
    m.setPositions(p)
    assert np.array_equal(m.returnPositions(), p)
    m.computeGeometry()
    assert np.array_equal(patched, m.areaPerimeter(), equal_nan=True)
    assert m.deviceStatus() == 0


def test_replayed_replicas_of_a_batch_match_oracle(svm_lib, oracle_mod):
    """Replicas that are replayed next to one that is not (150 cells)."""
    svm = svm_lib
    if svm.device_count() < 1:
        pytest.fail("no CUDA device: the GPU tests need a GB300")
    threshold = 0.2
    made = [crowded(svm, n, seed, edges) for n, seed, edges in ((400, 6, 300), (150, 7, 100), (1000, 8, 900))]
    topos = [t for t, _, _ in made]
    pos = [p.astype(np.float32).astype(np.float64) for _, p, _ in made]
    b = svm.sphericalVertexModelBatch([t.nCells for t in topos], None, topologies=topos)
    b.setT1Threshold(threshold)
    b.setPositions(np.concatenate(pos))
    b.enforceTopology()
    stats, got = b.t1Stats(), b.takeFlips()
    p, vn, vc = b.returnPositions(), b.vertexNeighbors(), b.vertexCellNeighbors()
    assert 1 <= stats["rollbacks"] <= 2, stats
    total = 0
    for r, (topo, _, R) in enumerate(made):
        om, flips = oracle_pass(oracle_mod, topo, pos[r], R, threshold)
        v, c = b.vertexSlice(r), b.cellSlice(r)
        mine = got[(got[:, 0] >= v.start) & (got[:, 0] < v.stop)]
        assert np.array_equal(mine - v.start, flips), r
        assert np.array_equal(vn[v] - v.start, om.vertex_neighbors()), r
        assert np.array_equal(vc[v] - c.start, om.vertex_cells()), r
        assert rel_err(p[v], om.positions(), R) < TOL["mixed"], r
        total += len(flips)
    assert stats["flips"] == total == len(got) and b.deviceStatus() == 0
