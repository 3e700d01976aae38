"""Data of more samples than a grid has blocks for: 65535 of 32."""
import numpy as np
import pytest

from cases import context
from fwi3d_b200 import lib, synth


@pytest.mark.gpu
def test_migration_of_more_than_65535_blocks_of_samples():
    n, dh, nt = 6, 10.0, 65535 * 32 + 33
    v = np.full((n, n, n), 2000.0, np.float32)
    src = np.array([[20.0, 20.0, 20.0]], np.float32)
    rec = np.array([[30.0, 10.0, 40.0], [10.0, 30.0, 10.0], [30.0, 10.0, 40.0]], np.float32)
    c = context(synth.Workload("long", n, n, n, dh, nt, 1e-3, 30.0, 4, v, src, rec), lib.BOUNDARY_RBC)
    c.set_velocity(v)
    # only beyond the first 65535 blocks, which is where the loop starts
    data = np.zeros((3, nt), np.float32)
    data[:, -33:] = 100.0 * np.random.default_rng(3).standard_normal((3, 33))
    c.rtm_shots([0], data)
    img, ill = c.get_accumulators()
    assert np.isfinite(img).all() and np.abs(img).max() > 0.0 and ill.max() > 0.0
