"""What a user of the spherical vertex model has it do, as cases that can be timed and compared.

Each case is one call, or one short loop, of the package's public classes (or of the C ABI where that
is the interface: the host-buffer step) on inputs made from a seed.  The sizes are those of the
project's workloads -- 200 cells, 20,000 cells, 100,000 cells, 1,000,000 cells, a batch of 512
replicas of 100 to 5,000 cells -- and odd ones between them.

Starting states are built here, not by running the dynamics: cell centres on a spherical Fibonacci
lattice moved by a seeded normal jitter, which gives a disordered, mostly hexagonal sheet with short
edges in it, so that the steps find T1 candidates as an equilibrated state does.  The state of a model
is its user's own: a step case goes on from where its last pass ended, as a simulation does.
"""
import ctypes
import math

import numpy as np
import torch

import curvedspacevertexmodel_gb300 as svm
from curvedspacevertexmodel_gb300 import _lib, warm_start

GOLDEN = math.pi * (3.0 - math.sqrt(5.0))
JITTER = 0.16           # of the lattice spacing
A0, T1_LENGTH, DT = 1.0, 0.04, 0.01


def listed():
    return [
        # The smallest simulation (200 cells, the reference's own default size): kernel latency and launches.
        {"name": "brownian_200", "kind": "brownian", "form": "fp64", "cells": 200, "steps": 16, "p0": 3.8, "T": 0.01},
        # The headline workload: overdamped dynamics of 100,000 cells in the plain FP64 form.
        {"name": "brownian_100k", "kind": "brownian", "form": "fp64", "cells": 100000, "steps": 4, "p0": 3.8, "T": 0.01},
        # The same sheet in the FP32-bulk / FP64-area form, as long runs use it.
        {"name": "mixed_100k", "kind": "brownian", "form": "mixed", "cells": 100000, "steps": 8, "p0": 3.8, "T": 0.01},
        # The largest single sphere.
        {"name": "mixed_1m", "kind": "brownian", "form": "mixed", "cells": 1000000, "steps": 4, "p0": 3.75, "T": 0.005},
        # A parameter sweep: uneven replicas stepped together.
        {"name": "batch_512", "kind": "batch", "replicas": 512, "smallest": 100, "largest": 5000, "steps": 4},
        # A quench: FIRE in the vector form with T1 flips, from the network's warm start.
        {"name": "fire_20k", "kind": "fire", "cells": 20000, "p0": 3.7, "iterations": 128, "warm": True, "t1": True},
        # A host program that owns the positions: upload, one step, download, energy.
        {"name": "host_step_100k", "kind": "host_step", "cells": 100000, "p0": 3.8, "T": 0.01},
        # One evaluation of energy and forces at given positions (an outside minimiser or sampler).
        {"name": "evaluate_5003", "kind": "evaluate", "form": "fp64", "cells": 5003, "p0": 3.85},
        # Setting up a sphere: the Voronoi topology of random cell centres.
        {"name": "topology_100k", "kind": "topology", "cells": 100000},
        # Self-propelled vertices with Vicsek alignment.
        {"name": "vicsek_20k", "kind": "vicsek", "cells": 20000, "p0": 3.8, "steps": 8},
        # Metric neighbour lists of a sphere's vertices, fetched to the host.
        {"name": "neighbours_20k", "kind": "neighbours", "points": 39996, "range": 1.0},
        # Training the warm start's network: one epoch of mini-batches.
        {"name": "train_64k", "kind": "train", "samples": 65537, "batch": 4096},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["brownian", "mixed", "mixed", "brownian", "batch", "fire", "host_step", "evaluate", "topology",
                       "vicsek", "neighbours", "train", "predict"])
    p0 = round(rng.uniform(3.6, 3.95), 3)
    T = round(math.exp(rng.uniform(math.log(1e-3), math.log(2e-2))), 5)
    if kind == "brownian":
        n = _log(rng, 100, 100000)
        return {"kind": "brownian", "form": "fp64", "cells": n, "steps": 4 if n > 30000 else rng.randint(3, 12), "p0": p0, "T": T}
    if kind == "mixed":
        n = _log(rng, 100, 1000000)
        return {"kind": "brownian", "form": "mixed", "cells": n, "steps": 4 if n > 100000 else rng.randint(3, 12), "p0": p0, "T": T}
    if kind == "batch":
        return {"kind": "batch", "replicas": _log(rng, 2, 500), "smallest": 100, "largest": _log(rng, 400, 5000),
                "steps": rng.randint(2, 4)}
    if kind == "fire":
        return {"kind": "fire", "cells": _log(rng, 200, 20000), "p0": round(rng.uniform(3.6, 3.8), 3),
                "iterations": rng.randint(32, 128), "warm": rng.random() < 0.5, "t1": rng.random() < 0.7}
    if kind == "host_step":
        return {"kind": "host_step", "cells": _log(rng, 200, 100000), "p0": p0, "T": T}
    if kind == "evaluate":
        return {"kind": "evaluate", "form": rng.choice(["fp64", "fp64_vector"]), "cells": _log(rng, 100, 20000), "p0": p0}
    if kind == "topology":
        return {"kind": "topology", "cells": _log(rng, 100, 100000)}
    if kind == "vicsek":
        return {"kind": "vicsek", "cells": _log(rng, 100, 20000), "p0": p0, "steps": rng.randint(2, 8)}
    if kind == "neighbours":
        return {"kind": "neighbours", "points": _log(rng, 300, 39000), "range": round(rng.uniform(0.6, 1.1), 3)}
    return {"kind": kind, "samples": _log(rng, 2000, 65000), "batch": rng.choice([512, 1000, 4096])}


# ---- inputs ----------------------------------------------------------------------------------------
def _sheet(cells, rng):
    """Cell centres: a spherical Fibonacci lattice with jitter, radius sqrt(cells / 4 pi)."""
    i = np.arange(cells) + 0.5
    z = 1.0 - 2.0 * i / cells
    s = np.sqrt(1.0 - z * z)
    p = np.stack([s * np.cos(GOLDEN * i), s * np.sin(GOLDEN * i), z], 1)
    p += rng.normal(0.0, JITTER * math.sqrt(4.0 * math.pi / cells), p.shape)
    return math.sqrt(cells / (4.0 * math.pi)) * p / np.linalg.norm(p, axis=1, keepdims=True)


def _noise(seed):
    n = svm.noiseSource()
    n.setReproducibleSeed(seed)
    return n


def _model(cells, p0, seed, form="fp64"):
    rng = np.random.default_rng([seed, cells])
    topo = svm.Topology(_sheet(cells, rng), device=True)
    m = svm.sphericalVertexModel(cells, _noise(seed % 100003), A0, p0, topology=topo)
    m.setT1Threshold(T1_LENGTH)
    if form != "fp64":
        m.precision = form
    return m


def _brownian(model, T, seed):
    bd = svm.brownianDynamics()
    bd.setModel(model)
    bd.setT(T)
    bd.setDeltaT(DT)
    bd.noise.setReproducibleSeed(seed % 100003 + 1)
    return bd


class _DeviceArray:
    """The model's positions on the device, where an analysis on the GPU reads them.  The tensor made of
    this object holds it, and with it the model whose memory it shows."""

    def __init__(self, model):
        self.model = model
        p = ctypes.c_void_p()
        _lib.call("svm_model_device_positions", model.handle, ctypes.byref(p))
        self.__cuda_array_interface__ = {"shape": (model.nVertices, 4), "data": (p.value, False), "version": 3,
                                         "typestr": "<f4" if model.precision == "mixed" else "<f8", "strides": None}


def _positions(model):
    return torch.as_tensor(_DeviceArray(model), device="cuda")[:, :3]


def _samples(case, seed):
    """Features and targets of the warm start's network: tangent-frame offsets of order one and a
    displacement that depends on them."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    n = case["samples"]
    X = torch.randn((n, 24), generator=g, device="cuda") * 0.7
    A = torch.randn((24, 2), generator=g, device="cuda") * 0.2
    Y = torch.tanh(X @ A) + 0.1 * torch.randn((n, 2), generator=g, device="cuda")
    return X, Y.contiguous()


def prepare(case, seed):
    kind = case["kind"]
    if kind == "brownian":
        m = _model(case["cells"], case["p0"], seed, case["form"])
        return {"case": case, "model": m, "updater": _brownian(m, case["T"], seed)}
    if kind == "batch":
        R = case["replicas"]
        sizes = np.random.default_rng([R, case["largest"]]).uniform(math.log(case["smallest"]), math.log(case["largest"]), R)
        sizes = np.exp(sizes).astype(int)  # the sweep's sizes are the case's; the spheres are the seed's
        rng = np.random.default_rng([seed, R])
        topos = [svm.Topology(_sheet(int(n), rng), device=True) for n in sizes]
        b = svm.sphericalVertexModelBatch(sizes, None, A0, rng.uniform(3.6, 3.95, R), topologies=topos)
        b.setT1Threshold(T1_LENGTH)
        b.setTemperatures(np.exp(rng.uniform(math.log(1e-4), math.log(1e-1), R)))
        return {"case": case, "model": b, "updater": _brownian(b, 0.0, seed)}
    if kind == "fire":
        m = _model(case["cells"], case["p0"], seed, "fp64_vector")
        m.restrictedMotion = not case["t1"]
        path = warm_start.__file__.rsplit("/", 1)[0] + "/data/warm_start_n20k.npz"
        net = warm_start.load(path)
        net.setOutputScale(0.25 * net.outputScale)
        return {"case": case, "model": m, "start": m.saveState(), "net": net, "rest": np.zeros((m.nVertices, 3))}
    if kind == "host_step":
        m = _model(case["cells"], case["p0"], seed)
        src = torch.from_numpy(m.returnPositions().reshape(-1)).pin_memory()
        return {"case": case, "model": m, "pos": [src, torch.empty_like(src).pin_memory()], "seed": seed % 100003}
    if kind == "evaluate":
        m = _model(case["cells"], case["p0"], seed, case["form"])
        return {"case": case, "model": m, "pos": m.returnPositions()}
    if kind == "topology":
        rng = np.random.default_rng([seed, case["cells"]])
        p = rng.normal(size=(case["cells"], 3))  # uniform on the sphere, as the reference draws its centres
        p *= math.sqrt(case["cells"] / (4.0 * math.pi)) / np.linalg.norm(p, axis=1, keepdims=True)
        return {"case": case, "centres": p}
    if kind == "vicsek":
        m = _model(case["cells"], case["p0"], seed)
        u = svm.sphericalVectorialVicsek()
        u.setModel(m)
        u.setDeltaT(DT)
        u.setV0(0.1)
        u.setEta(0.3)
        u.noise.setReproducibleSeed(seed % 100003 + 1)
        return {"case": case, "model": m, "updater": u}
    if kind == "neighbours":
        n = case["points"]
        rng = np.random.default_rng([seed, n])
        R = math.sqrt((n + 4) / 2 / (4.0 * math.pi))
        p = _sheet(n, rng)
        p *= R / np.linalg.norm(p, axis=1, keepdims=True)
        return {"case": case, "points": torch.from_numpy(np.ascontiguousarray(p)).cuda(),
                "list": svm.neighborList(case["range"], R + 2.5)}
    X, Y = _samples(case, seed)
    return {"case": case, "X": X, "Y": Y, "net": svm.warmStartNetwork(seed % 1009)}


# ---- one pass ---------------------------------------------------------------------------------------
def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind in ("brownian", "batch"):
        state["updater"].run(case["steps"])
        return _positions(state["model"])
    if kind == "fire":
        m = state["model"]
        m.loadState(state["start"])
        m.setVelocities(state["rest"])
        if case["warm"]:
            state["net"].warmStart(m)
        fire = svm.energyMinimizerFIRE(m)
        fire.setFIREParameters(*warm_start.FIRE_PARAMS)
        fire.setCriterion(_lib.SVM_FIRE_MAX_FORCE)
        fire.setMaximumIterations(case["iterations"])
        fire.minimize()
        return {"positions": m.returnPositions(), "energy": m.computeEnergy(), "neighbours": m.vertexNeighbors()}
    if kind == "host_step":
        src, dst = state["pos"]
        e = ctypes.c_double()
        _lib.call("svm_brownian_step_io", state["model"].handle, case["T"], DT, 1.0, state["seed"], src.numpy(), dst.numpy(),
                  ctypes.byref(e))
        state["pos"] = [dst, src]
        return {"positions": dst, "energy": e.value}
    if kind == "evaluate":
        m = state["model"]
        m.setPositions(state["pos"])
        m.computeForces()
        return {"energy": m.computeEnergy(), "forces": m.returnForces(), "area_perimeter": m.areaPerimeter()}
    if kind == "topology":
        t = svm.Topology(state["centres"], device=True)
        # (t.rings holds the same incidences cell by cell; its width is the largest ring's, the seed's)
        return [t.vertexPositions, t.ringCounts, t.vertexCells, t.vertexNeighbors]
    if kind == "vicsek":
        state["updater"].run(case["steps"])
        return {"positions": _positions(state["model"]), "directors": state["model"].returnDirectors()}
    if kind == "neighbours":
        nl = state["list"]
        nl.computeNeighborLists(state["points"])
        return [nl.neighborsPerParticle, nl.particleIndices, nl.neighborVectors, nl.neighborDistances]
    if kind == "train":
        losses = state["net"].train(state["X"], state["Y"], epochs=1, batch=case["batch"], lr=1e-3)
        return {"losses": losses, "weights": state["net"].weights()}
    return state["net"].predict(state["X"])


# ---- what a pass cannot do without --------------------------------------------------------------------
# Operations per vertex and step: the force in closed form (six triangle gradients of ~75 operations and
# three edge gradients of ~30), three included angles and 1.5 arcs of ~40, the move (~60); per FIRE
# iteration the vector form's ~400, the geometry, and the minimiser's own ~40.
_STEP_FLOPS = 6 * 75 + 3 * 30 + 5 * 40 + 60
_FIRE_FLOPS = 400 + 5 * 40 + 40
_MLP = 24 * 64 + 64 * 64 + 64 * 2


def work(case):
    kind = case["kind"]
    if kind == "train":
        return {"bytes": case["samples"] * 4.0 * (24 + 2 + 1), "flops": 6.0 * _MLP * case["samples"]}
    if kind == "predict":
        return {"bytes": case["samples"] * 4.0 * (24 + 2), "flops": 2.0 * _MLP * case["samples"]}
    if kind == "neighbours":
        per = 2.0 * (4.0 * math.pi * 0.25 * case["range"] ** 2)  # points in range at two per unit area
        return {"bytes": case["points"] * (24 + 4 + per * 36), "flops": case["points"] * per * 3 * 9}
    if kind == "batch":
        a, b = case["smallest"], case["largest"]
        cells = case["replicas"] * ((b - a) / math.log(b / a) if b > a else a)
    else:
        cells = case["cells"]
    nv = 2.0 * cells
    if kind == "topology":
        return {"bytes": cells * (24 + 8 * 4 + 4) + nv * (24 + 24), "flops": cells * 70 * 20.0}
    if kind == "fire":
        return {"bytes": nv * (24 * 2 + 36) + cells * 48, "flops": nv * _FIRE_FLOPS * case["iterations"]}
    real = 4 if kind == "batch" or case.get("form") == "mixed" else 8
    steps = case.get("steps", 1)
    out = 1 + (kind in ("vicsek",))
    return {"bytes": nv * (3 * real * (1 + out) + 36) + cells * 16, "flops": nv * _STEP_FLOPS * steps}


# ---- the same in 64 bits ------------------------------------------------------------------------------
def _exact_evaluate(case, seed):
    """Areas by the vertex-angle excess, perimeters, energy and its gradient, in numpy."""
    s = prepare(dict(case, form="fp64"), seed)
    m, pos, R = s["model"], s["pos"], s["model"].radius
    rings, counts = m.rings()
    n = counts.astype(int)
    c = np.repeat(np.arange(len(n)), n)
    k = np.arange(len(c)) - np.repeat(np.cumsum(n) - n, n)
    v, l, x = rings[c, k], rings[c, (k - 1) % n[c]], rings[c, (k + 1) % n[c]]
    P, r = pos[v], np.linalg.norm(pos[v], axis=1, keepdims=True)
    a = P / r

    def dot(p, q):
        return np.sum(p * q, axis=1, keepdims=True)

    def add(values, where, size):
        return np.stack([np.bincount(where, w, size) for w in values.T], 1)

    dl, dx = pos[l] - P, pos[x] - P
    # arcs from chords; angles between the tangents at the vertex, from successor to predecessor
    arc = 2.0 * R * np.arcsin(np.linalg.norm(dl, axis=1) / (2.0 * R))
    tl, tx = dl - dot(dl, a) * a, dx - dot(dx, a) * a
    turn = np.arctan2(np.sum(a * np.cross(tx, tl), axis=1), dot(tx, tl)[:, 0])
    angle = np.where(turn < 0, turn + 2 * np.pi, turn)
    if np.median(angle) > np.pi:
        angle = 2 * np.pi - angle
    area = (np.bincount(c, angle, len(n)) - (n - 2) * np.pi) * R * R
    per = np.bincount(c, arc, len(n))
    cen = add(P, c, len(n))
    cen *= R / np.linalg.norm(cen, axis=1, keepdims=True)
    dA, dP = (area - A0)[c][:, None], (per - case["p0"])[c][:, None]
    energy = float(np.sum((area - A0) ** 2 + (per - case["p0"]) ** 2))

    def geodesic(d):
        t = d - dot(d, a) * a
        return -t / np.linalg.norm(t, axis=1, keepdims=True)

    def triangle(b, g):  # gradient of the signed area of (v, v + b, v + g), from tan(E / 2) = N / D
        b, g = b / r, g / r
        bg = np.cross(b, g)
        bc = np.cross(a, g) + np.cross(b, a) + bg
        N, D = dot(a, bg), 4.0 - dot(b, b) - dot(g, g) + dot(b, g)
        w = 2.0 * (D * bc - N * (b + g)) / (N * N + D * D)
        return R * (w - dot(w, a) * a)

    dc = cen[c] - P
    f = -2.0 * dP * (geodesic(dl) + geodesic(dx)) - 2.0 * dA * (triangle(dl, dc) + triangle(dc, dx))
    return {"energy": energy, "forces": add(f, v, len(pos)), "area_perimeter": np.stack([area, per], 1)}


def _exact_network(case, seed):
    s = prepare(case, seed)
    X, Y = s["X"].double(), s["Y"].double()
    w = torch.from_numpy(s["net"].weights()).double().cuda()
    cut = [24 * 64, 64, 64 * 64, 64, 64 * 2, 2]

    def net(flat, x):
        W1, b1, W2, b2, W3, b3 = torch.split(flat, cut)
        h = torch.relu(x @ W1.view(64, 24).T + b1)
        h = torch.relu(h @ W2.view(64, 64).T + b2)
        return h @ W3.view(2, 64).T + b3

    def rounded(flat):
        return flat.float().bfloat16().double()

    if case["kind"] == "predict":
        return net(rounded(w), X)
    order = torch.from_numpy(np.random.default_rng(0).permutation(len(X))).cuda()
    m, v, total, step = torch.zeros_like(w), torch.zeros_like(w), 0.0, 0
    for first in range(0, len(X), case["batch"]):
        at = order[first:first + case["batch"]]
        q = rounded(w).requires_grad_()
        loss = (net(q, X[at]) - Y[at]).square().sum()
        g, = torch.autograd.grad(loss / len(at), q)
        total += float(loss)
        step += 1
        m = 0.9 * m + 0.1 * g
        v = 0.999 * v + 0.001 * g * g
        w = w - 1e-3 * (m / (1 - 0.9 ** step)) / ((v / (1 - 0.999 ** step)).sqrt() + 1e-8)
    return {"losses": [total / len(X)], "weights": w.cpu().numpy()}


def exact(case, seed):
    if case["kind"] == "evaluate":
        return _exact_evaluate(case, seed)
    if case["kind"] in ("train", "predict"):
        return _exact_network(case, seed)
    # the steps and the quench flip edges as they go: their states have no closed 64-bit restatement
    # that follows the same flips in a few seconds; topologies and lists are whole numbers first
    return None
