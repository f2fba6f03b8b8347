"""Runs of odd and even numbers of steps (a captured pair of steps per role of the position buffers) against the
same steps one by one, bit for bit, with the temperature and the threshold changed in between."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", ["fp64", "fp64_vector", "mixed"])
def test_runs_equal_single_steps(svm_lib, form):
    svm = svm_lib
    if svm.device_count() < 1:
        pytest.fail("no CUDA device: the GPU tests need a GB300")
    models = []
    for _ in range(2):
        noise = svm.noiseSource()
        noise.setReproducibleSeed(21)
        m = svm.sphericalVertexModel(150, noise, 1.0, 3.8)
        m.setT1Threshold(0.04)
        m.precision = form
        bd = svm.brownianDynamics()
        bd.setModel(m)
        bd.noise.setReproducibleSeed(4)
        models.append((m, bd))
    (a, run), (b, single) = models
    for steps, T, threshold in ((3, 0.01, 0.04), (5, 0.01, 0.04), (2, 0.01, 0.04), (3, 0.02, 0.04), (1, 0.02, 0.04),
                                (9, 0.02, 0.04), (3, 0.02, 0.08), (3, 0.02, 0.08), (7, 0.01, 0.08)):
        for m, bd in models:
            bd.setT(T)
            m.setT1Threshold(threshold)
        run.run(steps)
        for _ in range(steps):
            single.integrateEquationOfMotion()
        assert np.array_equal(a.returnPositions(), b.returnPositions())
        assert np.array_equal(a.vertexNeighbors(), b.vertexNeighbors())
    assert np.array_equal(a.takeFlips(), b.takeFlips())
