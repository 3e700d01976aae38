"""Blobs of the random pad: their number, order and place are those of a sampling
that makes every draw where it is used, however the draws are made ahead."""
import numpy as np
import pytest

from fwi3d_b200 import lib

# cells, pad and blob radius -> blobs of seeds 0..7, and over these seeds the sum of
# the mean of (1 + index) * (x + y + z)
KNOWN = [
    ((1, 4, 100.0), [1, 1, 1, 1, 1, 1, 1, 1], 1265.05997),
    ((6, 4, 50.0), [17, 19, 15, 18, 18, 18, 16, 16], 13428.4246),
    ((24, 8, 100.0), [41, 39, 36, 42, 39, 39, 40, 41], 89948.9477),
    ((60, 10, 100.0), [196, 189, 193, 190, 200, 196, 199, 199], 881901.262),
    ((24, 8, 30.0), [883, 895, 888, 888, 876, 876, 898, 883], 1932223.45),
    ((60, 20, 40.0), [5244, 5213, 5304, 5257, 5249, 5212, 5265, 5262], 28698307.2),
]


@pytest.mark.gpu
@pytest.mark.parametrize("pad,counts,total", KNOWN)
def test_points_of_a_pad(pad, counts, total):
    n, nb, ratio = pad
    ctx = lib.Context(n, n, n, nb, 10.0, 30, 1e-3, 30.0, lib.BOUNDARY_RBC)
    ctx.set_velocity(np.full((n, n, n), 2000.0, np.float32))
    got, s = [], 0.0
    for seed in range(8):
        b = np.asarray(ctx.random_boundary_recipe(kind=0, ratio=ratio, varVp=500.0, seed=seed)[2], np.float64).reshape(-1, 5)
        got.append(len(b))
        s += (b[:, :3] * np.arange(1, len(b) + 1)[:, None]).sum() / len(b)
    assert got == counts
    assert s == pytest.approx(total, rel=1e-6)  # (total has nine digits)
