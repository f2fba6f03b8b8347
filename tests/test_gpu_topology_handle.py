"""A device-built topology's handle (svm_topology_*), as a C caller keeps one: what it holds on the device."""
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
