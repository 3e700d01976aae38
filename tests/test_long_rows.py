"""Image and gradient post-processing of few and long z rows, which have a block
each, on both sides of that rule, against the FP64 oracle."""
import numpy as np
import pytest

import oracle as orc
from fwi3d_b200 import lib


@pytest.mark.gpu
@pytest.mark.parametrize("nz,nx,ny", [(64, 3, 5), (65, 3, 5), (255, 1, 1), (256, 2, 1), (257, 1, 3), (700, 4, 3),
                                      (66, 7, 169), (66, 37, 32)])
def test_post_processing(nz, nx, ny):
    import torch
    nb, dh, zmask = 4, 10.0, 35.0
    rng = np.random.default_rng(nz + nx)
    shape = (ny + 2 * nb, nx + 2 * nb, nz + 2 * nb)
    img, ill = rng.standard_normal(shape).astype(np.float32), rng.uniform(0.5, 2.0, shape).astype(np.float32)
    ctx = lib.Context(nz, nx, ny, nb, dh, 50, 1e-3, 30.0, lib.BOUNDARY_RBC)
    d_img, d_ill = torch.from_numpy(img).cuda(), torch.from_numpy(ill).cuda()
    torch.cuda.synchronize()
    ctx.set_accumulators_dev(d_img.data_ptr(), d_ill.data_ptr())
    want = orc.rtm_post(img, ill, nz, nx, ny, nb, dh)
    # three quotients and their difference in FP32: a few 2^-24 of the largest
    assert np.abs(ctx.rtm_image() - want).max() <= 1e-6 * np.abs(want).max()
    got, gmax = ctx.gradient_post(zmask)
    want, wmax = orc.gradient_post(img, ill, nz, nx, ny, nb, dh, zmask)
    assert np.abs(got - want).max() <= 2e-6 and abs(gmax - wmax) <= 1e-6 * wmax
