"""The copies between dense and pitched volumes and the post-processing, where
a warp takes a z row: rows just below, at and above one and four warp widths,
fewer rows than warps, and more than one pass of the grid."""
import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("nz,nx,ny", [(23, 4, 5), (24, 9, 4), (25, 7, 6), (120, 5, 3), (121, 6, 4), (13, 150, 170)])
def test_rows_of_every_length(nz, nx, ny):
    import torch
    from fwi3d_b200 import lib
    nb, dh = 4, 10.0
    rng = np.random.default_rng(nz)
    ctx = lib.Context(nz, nx, ny, nb, dh, 20, 1e-3, 30.0, lib.BOUNDARY_RBC)
    vp = (2000 + 500 * rng.random((ny, nx, nz))).astype(np.float32)
    ctx.set_velocity(vp)
    np.testing.assert_array_equal(ctx.get_padded_velocity(), np.pad(vp, nb, mode="edge"))

    shape = (ny + 2 * nb, nx + 2 * nb, nz + 2 * nb)
    img = rng.standard_normal(shape).astype(np.float32)
    ill = rng.uniform(0.5, 2.0, shape).astype(np.float32)
    ill[rng.random(shape) < 0.1] = 0.0
    d_img, d_ill = torch.from_numpy(img).cuda(), torch.from_numpy(ill).cuda()
    torch.cuda.synchronize()
    ctx.set_accumulators_dev(d_img.data_ptr(), d_ill.data_ptr())
    for got, want in zip(ctx.get_accumulators(), (img, ill)):
        np.testing.assert_array_equal(got, want)

    # the same FP32 operations in the same order; doubling and the sign are
    # exact, so only the last product may round once more or less
    q = np.divide(img, ill, out=np.zeros_like(img), where=ill != 0)[nb:-nb, nb:-nb, nb:-nb]
    want = np.zeros_like(q)
    want[:, :, 1:-1] = -(q[:, :, :-2] - 2 * q[:, :, 1:-1] + q[:, :, 2:]) * np.float32(1 / dh**2)
    np.testing.assert_allclose(ctx.rtm_image(), want, rtol=2.0**-22, atol=0)
    g, gmax = ctx.gradient_post(0.0)
    m = np.abs(want).max()
    assert abs(gmax - m) <= 2.0**-22 * m
    np.testing.assert_allclose(g, want / m, rtol=2.0**-20, atol=0)
