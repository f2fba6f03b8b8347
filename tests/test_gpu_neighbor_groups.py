"""The neighbour list's groups of threads at their edges: eight threads a point, 32 points a block,
four bins a thread in rounds of 32 bins, 32 candidates a thread at a time.  Against the oracle, bit
for bit (displacements and distances are the reference's FP64 expressions in its order)."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sub_grid", [1, 2, 3])            # 27, 117 and 311 bins in the mask or so
@pytest.mark.parametrize("n,crowd", [(1, 0), (31, 0), (32, 32), (33, 33), (65, 64), (257, 100), (1000, 0)])
def test_groups_match_oracle(svm_lib, n, crowd, sub_grid):
    import torch
    if svm_lib.device_count() < 1:
        pytest.fail("no CUDA device: the GPU tests need a GB300")
    rng = np.random.default_rng([n, crowd, sub_grid])
    radius, range_ = 2.5, 0.9                               # few bins a side: the mask crosses the faces
    pts = rng.uniform(-radius, radius, (n, 3))
    if crowd:                                               # up to 100 candidates in one or two bins
        pts[rng.permutation(n)[:crowd]] = 0.05 + rng.uniform(0.0, 0.3, (crowd, 3))
    nl = svm_lib.neighborList(range_, radius, sub_grid)
    for _ in range(2):                                      # the second call starts from the grown widths
        nl.computeNeighborLists(torch.from_numpy(pts.copy()).cuda())
        nm, npp, idx, vec, dist = oracle.neighbor_list(pts, range_, radius, sub_grid)
        assert nl.Nmax == nm
        assert np.array_equal(nl.neighborsPerParticle, npp)
        assert np.array_equal(nl.particleIndices, idx)
        assert np.array_equal(nl.neighborVectors, vec)
        assert np.array_equal(nl.neighborDistances, dist)
    nl.close()
