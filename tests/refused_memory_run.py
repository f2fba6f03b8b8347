"""Calls made again after the device memory they wanted was refused (tests/native/refuse_malloc.cpp, preloaded), each
against the same work done without a refusal.  Used by tests/test_gpu_refused_memory.py, which names the check."""
import ctypes as C
import json
import os
import sys

import numpy as np

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
for d in (os.path.join(ROOT, "tests"), os.path.join(ROOT, "oracle"), ROOT):
    sys.path.insert(0, d)
import curvedspacevertexmodel_gb300 as svm  # noqa: E402
import oracle  # noqa: E402
from curvedspacevertexmodel_gb300 import _lib  # noqa: E402
from test_gpu_t1_rollback import crowded, oracle_pass  # noqa: E402

shim = C.CDLL(os.environ["LD_PRELOAD"])
refuse_from, refused = C.c_size_t.in_dll(shim, "refuse_from"), C.c_int.in_dll(shim, "refused")


def refused_call(f):
    refuse_from.value, refused.value = 1, 0
    try:
        f()
        ok = False
    except _lib.SVMError:
        ok = refused.value > 0
    refuse_from.value = 0
    return ok


def wants_room(n, seed, edges, threshold, blocks):
    """A crowded sheet whose rings are to grow before its next T1 pass."""
    topo, pos, R = crowded(svm, n, seed, edges)
    m = svm.sphericalVertexModel(n, topology=topo, radius=R)
    m.setT1Threshold(threshold)
    m.setT1Blocks(blocks)
    m.setPositions(pos)
    m.setRingHeadroom(16)
    return m, topo, pos, R


def growth(blocks):
    """A T1 pass by itself, and a step, whose ring growth is refused once."""
    args = (400, 6, 300, 0.2, blocks)
    m, topo, pos, R = wants_room(*args)
    om, flips = oracle_pass(oracle, topo, pos, R, 0.2)
    rep = dict(refused=[refused_call(m.enforceTopology), refused_call(m.enforceTopology)])
    m.enforceTopology()
    rep["flips"] = np.array_equal(m.takeFlips(), flips) and len(flips) > 100
    rep["neighbours"] = np.array_equal(m.vertexNeighbors(), om.vertex_neighbors())
    rep["growths"], rep["status"] = m.ringInfo()["growths"], m.deviceStatus()
    # the refused step moved the vertices and left their flips to the next, as a restricted step does
    models = []
    for again in (True, False):
        m = wants_room(*args)[0]
        bd = svm.brownianDynamics()
        bd.setModel(m)
        bd.setT(0.0)
        bd.setDeltaT(1e-12)
        if again:
            rep["refused"].append(refused_call(bd.integrateEquationOfMotion))
        else:
            m.restrictedMotion = True
            bd.integrateEquationOfMotion()
            m.restrictedMotion = False
        bd.integrateEquationOfMotion()
        m.computeGeometry()
        models.append(m)
    a, b = models
    rep["step"] = (np.array_equal(a.returnPositions(), b.returnPositions()) and a.takeFlips().size > 0
                   and np.array_equal(a.vertexNeighbors(), b.vertexNeighbors())
                   and np.array_equal(a.areaPerimeter(), b.areaPerimeter(), equal_nan=True))
    rep["status"] |= a.deviceStatus() | b.deviceStatus()
    return rep


def train(first, refused_samples):
    """Two epochs of batches of 512 after a training call whose gradient sums found no room (and, with `first`, after an
    epoch before it): losses and weights as without that call."""
    import torch
    g = torch.Generator(device="cuda")
    g.manual_seed(3)
    n = max(2000, refused_samples)
    X, Y = torch.randn((n, 24), generator=g, device="cuda"), torch.randn((n, 2), generator=g, device="cuda")
    order = torch.arange(n, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()

    def epoch(net, samples, batch):
        loss = C.c_double()
        _lib.call("svm_mlp_train", net._h, C.c_void_p(X.data_ptr()), C.c_void_p(Y.data_ptr()), C.c_void_p(order.data_ptr()),
                  samples, batch, C.c_float(1e-3), C.byref(loss))
        return loss.value

    rep, results = {}, []
    for again in (False, True):
        net = svm.warmStartNetwork(7)
        losses = [epoch(net, 2000, 512)] if first else []
        if again:
            rep["refused"] = refused_call(lambda: epoch(net, refused_samples, refused_samples))
        losses += [epoch(net, 2000, 512) for _ in range(2)]
        results.append((losses, net.weights()))
    rep["losses"] = results[0][0] == results[1][0]
    rep["weights"] = bool(np.array_equal(results[0][1], results[1][1]))
    return rep


def lists(slots):
    """A neighbour list whose bins (2 slots) or rows (64 slots: bins that hold all) are to grow, refused once."""
    import torch
    rng = np.random.default_rng(5)
    p = rng.normal(size=(3000, 3))
    p *= 8.0 / np.linalg.norm(p, axis=1)[:, None]
    points = torch.from_numpy(p).cuda()
    rep, results = {}, []
    for again in (False, True):
        nl = svm.neighborList(1.0, 10.5, slotCapacity=slots)
        nl._ensure(len(p))
        if again:
            rep["refused"] = [refused_call(lambda: nl.computeNeighborLists(points)) for _ in range(2)]
        nl.computeNeighborLists(points)
        results.append((nl.neighborsPerParticle, nl.particleIndices, nl.neighborVectors, nl.neighborDistances))
    rep["longest"] = int(results[0][0].max())
    rep["same"] = all(a.shape == b.shape and np.array_equal(a, b) for a, b in zip(*results))
    return rep


if __name__ == "__main__":
    print(json.dumps({"growth": growth, "train": train, "lists": lists}[sys.argv[1]](*map(int, sys.argv[2:]))), flush=True)
