"""The blob pass of the random pad on its bricks, and the check of velocity
models, against their NumPy restatements."""
import numpy as np
import pytest

import rbc_oracle as ro
from fwi3d_b200 import lib, synth


def _ctx(n, nb):
    w = synth.small_case(n=n, nb=nb, nt=20, seed=6)
    ctx = lib.Context(w.nz, w.nx, w.ny, w.nb, w.dh, w.nt, w.dt, w.fmax, lib.BOUNDARY_RBC)
    ctx.set_velocity(w.vp)
    return w, ctx, ctx.get_padded_velocity()


@pytest.mark.gpu
@pytest.mark.parametrize("n,nb,ratio", [(40, 20, 12.0), (40, 20, 90.0), (21, 6, 15.0), ((70, 250, 260), 20, 60.0)])
def test_blob_pass_on_bricks(n, nb, ratio):
    """Bricks with more blobs than their list holds (small radii), with blobs
    that reach every brick, ragged last bricks, and the large bricks of grids
    that fill the GPU."""
    nz, nx, ny = n if isinstance(n, tuple) else (n, n + 3, n + 1)
    rng = np.random.default_rng(8)
    vp = (2000 + 500 * rng.random((ny, nx, nz))).astype(np.float32)
    ctx = lib.Context(nz, nx, ny, nb, 10.0, 20, 1e-3, 30.0, lib.BOUNDARY_RBC)
    ctx.set_velocity(vp)
    clean = ctx.get_padded_velocity()
    rbc = dict(kind=0, ratio=ratio, varVp=300.0)
    ctx.apply_random_boundary(seed=5, **rbc)
    got = ctx.get_padded_velocity()
    vlo, vhi, blobs = ctx.random_boundary_recipe(seed=5, **rbc)
    bg = ro.background(clean, nb, 0, ratio, 300.0, vlo, vhi, 5)
    want = ro.blob_pass(bg, nb, 10.0, blobs, vlo, vhi)
    d = np.abs(got.astype(np.float64) - want)
    # expf within 2 ulp and a few FP32 roundings of values below 4096 (ulp
    # 2.4e-4 m/s) per blob, some hundred blobs a cell at random signs; a cell
    # at 5 r may fall on either side (amp e^-12.5 = 1e-3 m/s)
    assert d.max() < 1e-2 and np.count_nonzero(d > 2e-3) <= 1e-4 * d.size
    assert np.abs(got - bg).max() > 50.0


@pytest.mark.gpu
@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf, -1.0, 0.0, -0.0])
@pytest.mark.parametrize("padded", [False, True])
def test_bad_velocities_are_refused_and_named(bad, padded):
    w, ctx, clean = _ctx(n=12, nb=5)
    put = ctx.set_padded_velocity if padded else ctx.set_velocity
    v = (clean if padded else w.vp).copy()
    for at in ([0], [v.size - 1], [v.size // 2, 7]):
        u = v.copy()
        u.reshape(-1)[at] = bad
        with pytest.raises(lib.FwiError) as e:
            put(u)
        assert e.value.code == 7 and f"velocity[{min(at)}]" in str(e.value)
        assert np.array_equal(ctx.get_padded_velocity(), clean)
    put(v)
    assert np.array_equal(ctx.get_padded_velocity(), clean)
