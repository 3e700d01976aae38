"""FP64 reductions on device buffers: sizes around the quads, blocks and rounds of
the kernels, with and without 16-byte alignment."""
import numpy as np
import pytest

from fwi3d_b200 import lib

pytestmark = pytest.mark.gpu

# one block sums 4 quads of each of its 256 threads a round; 888 blocks at most
ROUND = 4 * 4 * 256


@pytest.mark.parametrize("n", [1, 3, 4, 5, ROUND - 1, ROUND, ROUND + 1, 888 * ROUND - 1, 888 * ROUND + 5,
                               2 * 888 * ROUND + 3])
@pytest.mark.parametrize("offset", [0, 1])
def test_residual_and_dot(n, offset):
    import torch
    g = torch.Generator(device="cuda").manual_seed(n)
    a, b = (torch.randn(n + 1, generator=g, device="cuda")[offset:offset + n] for _ in range(2))
    res = torch.full((n + 2,), 7.0, device="cuda")
    with lib.Context(8, 8, 8, 4, 10.0, 8, 1e-3, 30.0) as ctx:
        torch.cuda.synchronize()
        got = ctx.residual_dev(a.data_ptr(), b.data_ptr(), n, res.data_ptr() + 4 * offset)
        again = ctx.residual_dev(a.data_ptr(), b.data_ptr(), n)
        dot = ctx.dot_dev(a.data_ptr(), b.data_ptr(), n)
    r = (a - b).cpu().numpy()
    kept = res.cpu().numpy()
    assert np.array_equal(kept[offset:offset + n], r)
    assert (kept[:offset] == 7.0).all() and (kept[offset + n:] == 7.0).all()
    # n products rounded to 53 bits: at most n * 2^-53 of the sum of magnitudes
    tol = max(n, 4) * 2.0 ** -53
    want = np.sum(r.astype(np.longdouble) ** 2)
    assert abs(got - want) <= tol * want and again == got
    p = a.cpu().numpy().astype(np.longdouble) * b.cpu().numpy()
    assert abs(dot - np.sum(p)) <= tol * np.sum(np.abs(p))
