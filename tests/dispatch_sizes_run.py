"""Three Brownian steps of a jittered sheet of each given number of cells, on the device and on the CPU
oracle with the same portable arccosine (as portable_acos_run.py): prints one JSON list of the
differences found.  Used by tests/test_gpu_dispatch_sizes.py.

    SVM_LIBRARY=.../libsvm_pacos.so python tests/dispatch_sizes_run.py JITTER T1_THRESHOLD 1501 1502 ...
"""
import json
import math
import sys

import numpy as np

from portable_acos_run import compare, oracle, svm


def sheet(cells, seed, jitter):
    """A spherical Fibonacci lattice with a normal jitter, in units of the cells' spacing."""
    rng = np.random.default_rng([seed, cells])
    i = np.arange(cells) + 0.5
    z = 1.0 - 2.0 * i / cells
    a = math.pi * (3.0 - math.sqrt(5.0)) * i
    p = np.stack([np.sqrt(1.0 - z * z) * np.cos(a), np.sqrt(1.0 - z * z) * np.sin(a), z], 1)
    p += rng.normal(0.0, jitter * math.sqrt(4.0 * math.pi / cells), p.shape)
    return math.sqrt(cells / (4.0 * math.pi)) * p / np.linalg.norm(p, axis=1, keepdims=True)


def run(cells, jitter, threshold, steps=3):
    topo = svm.Topology(sheet(cells, 3, jitter), device=True)
    m = svm.sphericalVertexModel(cells, svm.noiseSource(), 1.0, 3.8, topology=topo)
    m.setT1Threshold(threshold)
    rings, counts = m.rings(16)
    om = oracle.OracleModel(m.returnPositions(), rings, counts, m.vertexCellNeighbors(), m.vertexNeighbors(), m.radius)
    om.set_preferred(1.0, 3.8)
    om.set_t1_threshold(threshold)
    bd = svm.brownianDynamics()
    bd.setModel(m)
    bd.setT(0.01)
    noise = oracle.OracleNoise(cells)
    rep = dict(cells=cells, steps=0, checks=0, pos_bits_differ=0, flips_differ=0, topology_differ=0,
               area_perimeter_bits_differ=0, energy_cpu_order_bits_differ=0, energy_reduction_rel=0.0, flips=0)
    for _ in range(steps):
        xi = noise.normals(3 * m.nVertices)
        bd.injectNoise(xi)
        bd.integrateEquationOfMotion()
        om.brownian_step_noise(xi, 0.01, 0.01, 1.0)
        rep["flips"] += len(om.flips(clear=False))
        compare(m, om, rep, 1.0, (1.0, 3.8), True)
    m.computeForces()
    om.compute_forces()
    f, g = m.returnForces(), om.forces()
    rep["force_bits_differ"] = int(np.count_nonzero(f.view(np.uint64) != np.ascontiguousarray(g).view(np.uint64)))
    rep["status"] = m.deviceStatus()
    return rep


if __name__ == "__main__":
    oracle.set_portable_acos(True)
    print(json.dumps([run(int(n), float(sys.argv[1]), float(sys.argv[2])) for n in sys.argv[3:]]), flush=True)
