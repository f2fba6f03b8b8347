"""The warm-start network's kernels at the edges of their tiles (32 samples) and clusters (128 samples)
against the CPU reference (oracle/mlp.py), with the tolerances of test_gpu_mlp.py: FP32 chains of up to
64 products forward, of up to n products in the gradient."""
import numpy as np
import pytest

import mlp

pytestmark = pytest.mark.gpu
SIZES = [1, 31, 32, 33, 127, 128, 129, 257, 20000]


def _net(svm_lib, seed):
    net = svm_lib.warmStartNetwork(seed)
    w = np.random.default_rng(seed).normal(0, 0.25, net.parameterCount).astype(np.float32)
    net.setWeights(w)
    return net, w


def _data(n):
    rng = np.random.default_rng(n)
    return rng.normal(0, 1, (n, 24)).astype(np.float32), rng.normal(0, 1, (n, 2)).astype(np.float32)


@pytest.mark.parametrize("n", SIZES)
def test_predict_and_gradient(svm_lib, n):
    import torch
    net, w = _net(svm_lib, 6)
    X, T = _data(n)
    Xd, Td = torch.from_numpy(X).cuda(), torch.from_numpy(T).cuda()
    y, _ = mlp.forward(mlp.bf16(w), X.astype(np.float64))
    assert np.max(np.abs(net.predict(Xd).cpu().numpy() - y)) < 1e-4 * max(1.0, np.max(np.abs(y)))
    loss, g = net.gradient(Xd, Td)
    lref, gref = mlp.loss_and_grad(mlp.bf16(w), X.astype(np.float64), T.astype(np.float64))
    assert abs(loss - lref) < 1e-5 * lref
    assert np.linalg.norm(g - gref) < 1e-4 * np.linalg.norm(gref)


@pytest.mark.parametrize("n,batch", [(1, 8), (130, 129), (300, 128), (257, 1000)])
def test_epoch_loss_and_untouched_weights_at_rate_zero(svm_lib, n, batch):
    import torch
    net, w = _net(svm_lib, 7)
    X, T = _data(n)
    loss = net.train(torch.from_numpy(X).cuda(), torch.from_numpy(T).cuda(), epochs=1, batch=batch, lr=0.0)[0]
    lref, _ = mlp.loss_and_grad(mlp.bf16(w), X.astype(np.float64), T.astype(np.float64))
    assert abs(loss - lref) < 1e-5 * lref
    assert np.array_equal(net.weights(), w)
