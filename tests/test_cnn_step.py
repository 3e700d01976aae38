"""Two training steps of the preconditioner against a NumPy restatement of Adam
on the gradients that the steps return."""
import numpy as np
import pytest

from fwi3d_b200 import lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(20, 12, 10), (3, 2, 1)])
def test_weights_after_two_steps(shape):
    import torch
    nz, nx, ny = shape
    g = torch.Generator(device="cuda").manual_seed(4)
    x = torch.randn(3, ny, nx, nz, generator=g, device="cuda")
    y = torch.randn(ny, nx, nz, generator=g, device="cuda")
    torch.cuda.synchronize()
    net, lr = lib.Cnn(3), 1e-2
    w, b = (a.astype(np.float64) for a in net.get_weights())
    m, v = [np.zeros_like(w), np.zeros_like(b)], [np.zeros_like(w), np.zeros_like(b)]
    for step in (1, 2):
        _, gw, gb = net.train_step(shape, x.data_ptr(), y.data_ptr(), lr, want_grads=True)
        for k, (p, grad) in enumerate(((w, gw), (b, gb))):
            grad = grad.astype(np.float64)
            m[k] = 0.9 * m[k] + 0.1 * grad
            v[k] = 0.999 * v[k] + 0.001 * grad ** 2
            p -= lr * (m[k] / (1 - 0.9 ** step)) / (np.sqrt(v[k] / (1 - 0.999 ** step)) + 1e-8)
        got = net.get_weights()
        # an update is at most about lr, computed in a dozen FP32 roundings, of
        # which 1 - 0.999^step loses the most: 0.001 is 1.7e4 units of 2^-24
        for a, want in zip(got, (w, b)):
            assert np.abs(a - want).max() <= 2e-4 * lr
    # without a learning rate the weights stay
    net.train_step(shape, x.data_ptr(), y.data_ptr(), 0.0)
    for a, c in zip(net.get_weights(), got):
        assert np.array_equal(a, c)
