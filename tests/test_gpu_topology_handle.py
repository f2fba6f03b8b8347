"""A device-built topology's handle (svm_topology_*), as a C caller keeps one: what it holds on the device, and what the
calls on it wait for."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def centres(n):
    """A jittered spherical Fibonacci lattice of unit density."""
    rng = np.random.default_rng(n)
    i = np.arange(n) + 0.5
    z = 1 - 2 * i / n
    s, phi = np.sqrt(1 - z * z), np.pi * (3 - np.sqrt(5)) * i
    p = np.stack([s * np.cos(phi), s * np.sin(phi), z], 1) + rng.normal(0, 0.1 * np.sqrt(4 * np.pi / n), (n, 3))
    return np.sqrt(n / (4 * np.pi)) * p / np.linalg.norm(p, axis=1, keepdims=True)


def build(svm, pts):
    from curvedspacevertexmodel_gb300 import _lib
    h = C.c_void_p()
    _lib.call("svm_topology_from_points_gpu", np.ascontiguousarray(pts).reshape(-1), len(pts), None, C.byref(h))
    return h


def test_handle_holds_its_results_only(svm_lib):
    import torch
    from curvedspacevertexmodel_gb300 import _lib
    svm = svm_lib
    if svm.device_count() < 1:
        pytest.fail("no CUDA device: the GPU tests need a GB300")
    n = 200000
    pts = centres(n)
    _lib.lib().svm_topology_free(build(svm, pts))   # (the kernels are loaded from here on)
    before = torch.cuda.mem_get_info()[0]
    h = build(svm, pts)
    held = before - torch.cuda.mem_get_info()[0]
    nc, nv, w = C.c_int(), C.c_int(), C.c_int()
    _lib.call("svm_topology_sizes", h, C.byref(nc), C.byref(nv), C.byref(w))
    _lib.lib().svm_topology_free(h)
    results = 8 * 3 * nv.value + 4 * (2 * 3 * nv.value + n + n * w.value)
    assert held <= results + (8 << 20), (held, results)   # (the driver hands memory out in pages of 2 MB)
    assert before - torch.cuda.mem_get_info()[0] <= 0


def fetch(h):
    from curvedspacevertexmodel_gb300 import _lib
    nc, nv, w = C.c_int(), C.c_int(), C.c_int()
    _lib.call("svm_topology_sizes", h, C.byref(nc), C.byref(nv), C.byref(w))
    out = [np.empty(3 * nv.value), np.empty(nc.value * (w.value + 3), np.int32), np.empty(nc.value, np.uint32),
           np.empty(3 * nv.value, np.int32), np.empty(3 * nv.value, np.int32)]
    _lib.call("svm_topology_get", h, out[0], out[1], w.value + 3, out[2], out[3], out[4])
    return out


def host(svm, pts):
    """The arrays of the host's hull, in rows three entries wider than its rings."""
    t = svm.Topology(pts)
    rows = np.full((len(pts), t.rings.shape[1] + 3), -1, np.int32)
    for c, k in enumerate(t.ringCounts):
        rows[c, :k] = t.rings[c, :k]
    return [t.vertexPositions.reshape(-1), rows.reshape(-1), t.ringCounts, t.vertexCells.reshape(-1), t.vertexNeighbors.reshape(-1)]


def same(a, b):
    return all(np.array_equal(x, y) for x, y in zip(a, b))


def test_fetched_while_another_thread_captures(svm_lib):
    """Fetching and freeing a handle takes no part in a capture that another thread has under way, whatever its mode."""
    import threading
    import torch
    from curvedspacevertexmodel_gb300 import _lib
    svm = svm_lib
    if svm.device_count() < 1:
        pytest.fail("no CUDA device: the GPU tests need a GB300")
    pts = centres(500)
    h, expect, got = build(svm, pts), host(svm, pts), []

    def other():
        try:
            got.append(fetch(h))
            _lib.lib().svm_topology_free(h)
        except Exception as e:
            got.append(e)

    x = torch.zeros(1000, device="cuda")
    x += 1
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, capture_error_mode="global"):
        x += 1
        t = threading.Thread(target=other)
        t.start()
        t.join()
        x += 1
    g.replay()
    torch.cuda.synchronize()
    assert float(x[0]) == 3.0 and float(x[-1]) == 3.0
    assert len(got) == 1 and not isinstance(got[0], Exception), got
    assert same(got[0], expect)


def test_fetched_while_the_device_is_busy(svm_lib):
    """Fetching does not wait for work on the default stream."""
    import torch
    from curvedspacevertexmodel_gb300 import _lib
    svm = svm_lib
    if svm.device_count() < 1:
        pytest.fail("no CUDA device: the GPU tests need a GB300")
    pts = centres(500)
    h, expect = build(svm, pts), host(svm, pts)
    fetch(h)
    done = torch.cuda.Event()
    torch.cuda._sleep(1000)
    torch.cuda.synchronize()
    torch.cuda._sleep(1 << 30)   # half a second
    done.record()
    got = fetch(h)
    early = not done.query()
    torch.cuda.synchronize()
    _lib.lib().svm_topology_free(h)
    assert early and same(got, expect)


@pytest.mark.parametrize("spokes", [15, 16, 17, 24])
def test_rings_wider_than_the_rows_made_ahead(svm_lib, spokes):
    """A centre with up to 24 neighbours: rows of 16 entries are allocated before the rings are known."""
    from curvedspacevertexmodel_gb300 import _lib
    svm = svm_lib
    if svm.device_count() < 1:
        pytest.fail("no CUDA device: the GPU tests need a GB300")
    rng = np.random.default_rng(spokes)
    theta = np.concatenate([[0.0], 0.8 + 0.01 * rng.standard_normal(spokes), np.arccos(rng.uniform(-1, np.cos(1.2), 60))])
    phi = np.concatenate([[0.0], 2 * np.pi * (np.arange(spokes) + 0.2 * rng.random(spokes)) / spokes, rng.uniform(0, 2 * np.pi, 60)])
    pts = 2.5 * np.stack([np.sin(theta) * np.cos(phi), np.sin(theta) * np.sin(phi), np.cos(theta)], 1)
    h, expect = build(svm, pts), host(svm, pts)
    assert int(expect[2][0]) == expect[2].max() == spokes
    assert same(fetch(h), expect)
    _lib.lib().svm_topology_free(h)
