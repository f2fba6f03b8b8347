"""FIRE stops where its loop stops (energyMinimizerFIRE.cpp:186-196): a minimisation that ends within a batch of
launched iterations leaves the state of its last iteration, also while edges below the T1 threshold are left.
Compared with the same number of single iterations through the per-phase entry points, bit for bit."""
import numpy as np
import pytest

from gpu_helpers import load_gold

pytestmark = pytest.mark.gpu


def sheet(svm, n, form):
    noise = svm.noiseSource()
    noise.setReproducibleSeed(12)
    m = svm.sphericalVertexModel(n, noise, 1.0, 3.8)   # random centres: many short edges
    m.precision = form
    m.setT1Threshold(0.25)
    return m


def minimizer(svm, m, iterations):
    p = load_gold()["fire_params"]
    f = svm.energyMinimizerFIRE(m)
    f.setFIREParameters(p[0], p[1], p[2], p[3], p[4], p[5], int(p[6]), 1e-300, p[8])
    f.setMaximumIterations(iterations)
    return f


@pytest.mark.parametrize("iterations", [1, 5, 33, 40])
@pytest.mark.parametrize("cells,form", [(300, "fp64"), (300, "fp64_vector"), (25200, "fp64_vector")])
def test_minimize_ends_with_its_last_iteration(svm_lib, cells, form, iterations):
    svm = svm_lib
    if svm.device_count() < 1:
        pytest.fail("no CUDA device: the GPU tests need a GB300")
    a, b = sheet(svm, cells, form), sheet(svm, cells, form)
    fa, fb = minimizer(svm, a, iterations), minimizer(svm, b, iterations)
    fa.minimize()
    b.computeForces()
    for _ in range(iterations):
        fb.integrateEquationOfMotion()
        fb.fireStep()
    assert fa.getCurrentIterations() == iterations
    flips = b.takeFlips()
    assert np.array_equal(a.takeFlips(), flips) and len(flips) > 10
    assert np.array_equal(a.vertexNeighbors(), b.vertexNeighbors())
    assert np.array_equal(a.returnPositions(), b.returnPositions(), equal_nan=True)
    assert np.array_equal(a.returnForces(), b.returnForces(), equal_nan=True)
    assert np.array_equal(a.areaPerimeter(), b.areaPerimeter(), equal_nan=True)
    assert np.isfinite(a.returnPositions()).all()
    # the device still holds the stopped state's geometry and goes on from it as the other does
    assert a.computeEnergy() == b.computeEnergy()
    for m in (a, b):
        m.computeForces()
    assert np.array_equal(a.returnForces(), b.returnForces(), equal_nan=True)
    assert a.deviceStatus() == b.deviceStatus()
