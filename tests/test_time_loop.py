"""The one-launch time loops at the edges of their tiles and of their ticket
order, against the FP64 oracle with the FP32 bounds of tests/cases.py."""
import numpy as np
import pytest

import oracle as orc
from cases import TOL_GRAD, TOL_IMAGE, TOL_SEIS, context, indices, interior, oracle_wavelet, rel_l2
from fwi3d_b200 import lib, synth


def _workload(nz, nx, ny, nb, nt=70, nsrc=1, seed=0):
    """Random velocities; receivers in every x row of two depths, three of them
    on one cell, so that a plane of a column has more of them than a warp."""
    rng = np.random.default_rng(seed)
    dh = 10.0
    v = (1800 + 600 * rng.random((ny, nx, nz))).astype(np.float32)
    src = np.stack([(0.2 + 0.6 * rng.random(nsrc)) * (n - 1) * dh for n in (nx, ny, nz)], 1)
    xs, ys = np.arange(nx) * dh, np.arange(0, ny, 2) * dh
    rec = np.concatenate([synth.surface_grid(xs, ys, z * dh) for z in sorted({0, nz // 2})])
    rec = np.concatenate([rec, rec[:1], rec[:1]])
    return synth.Workload("loop", nz, nx, ny, dh, nt, 1e-3, 60.0, nb, v, src.astype(np.float32), rec,
                          abc_factor=0.02)


# (1, 1, 1) is the smallest grid; the others are one cell below, at and above
# tile sizes along z and x, with few and with many y planes
GRIDS = [(1, 1, 1, 4), (64, 8, 3, 4), (65, 9, 30, 4), (47, 40, 12, 6), (150, 25, 9, 5), (98, 15, 17, 7)]


@pytest.mark.gpu
@pytest.mark.parametrize("grid", GRIDS)
def test_forward_and_backward_match_the_oracle_on_every_tile(grid):
    w = _workload(*grid)
    src, rec = indices(w, w.nb)
    data = np.random.default_rng(1).standard_normal((len(w.rec), w.nt)).astype(np.float32)
    abc, rtm = context(w, lib.BOUNDARY_ABC), context(w, lib.BOUNDARY_RBC)
    grads = {dy: context(w, lib.BOUNDARY_RBC, flags=lib.FLAG_SUBTRACT_SOURCE | (lib.FLAG_GRAD_DY if dy else 0))
             for dy in (False, True)}
    for c in (abc, rtm, *grads.values()):
        c.set_velocity(w.vp)
    vpp = abc.get_padded_velocity()
    w64, _ = oracle_wavelet(abc, w)
    ref_abc = orc.forward(vpp, w.dh, w.dt, w.nt, abc.tlag, w64, src[0], rec, abc=True, nb=w.nb, factor=w.abc_factor)[0]
    ref_rbc, P, Q = orc.forward(vpp, w.dh, w.dt, w.nt, abc.tlag, w64, src[0], rec)
    ref = {}
    for mode, dy in ((0, False), (1, False), (1, True)):
        ref[mode, dy] = orc.backward(vpp, w.dh, w.dt, w.nt, abc.tlag, rec, data, P.copy(), Q.copy(), mode=mode,
                                     with_dy=dy, subtract_src=mode == 1, w=w64, src=src[0])[:2]
    for tile in range(-1, len(lib.tile_table())):
        for c in (abc, rtm, *grads.values()):
            c.set_tiles(tile, tile)
        assert rel_l2(abc.model_shots([0])[0], ref_abc) < TOL_SEIS, tile
        assert rel_l2(rtm.model_shots([0])[0], ref_rbc) < TOL_SEIS, tile
        for (mode, dy), (rimg, rill) in ref.items():
            c = grads[dy] if mode else rtm
            c.reset_accumulators()
            (c.gradient_shots if mode else c.rtm_shots)([0], data)
            img, ill = c.get_accumulators()
            e = [rel_l2(interior(a, w.nb), interior(b, w.nb)) for a, b in ((img, rimg), (ill, rill))]
            assert e[0] < (TOL_GRAD if mode else TOL_IMAGE) and e[1] < TOL_IMAGE, (tile, mode, dy, e)


@pytest.mark.gpu
@pytest.mark.parametrize("batch,shots", [(2, 5), (5, 5), (7, 6)])
def test_interleaved_shots_equal_single_shots(batch, shots):
    """Shots side by side in the ticket order, and a last batch that does not
    fill its slots."""
    w = _workload(30, 26, 22, 6, nsrc=shots, seed=3)
    single, many = context(w, lib.BOUNDARY_RBC), context(w, lib.BOUNDARY_RBC, max_batch=batch)
    for c in (single, many):
        c.set_velocity(w.vp)
    ids = list(range(shots))
    for a, b in zip(single.model_shots(ids), many.model_shots(ids)):
        assert np.array_equal(a, b)
    data = np.random.default_rng(2).standard_normal((shots * len(w.rec), w.nt)).astype(np.float32)
    for c in (single, many):
        c.rtm_shots(ids, data)
    for a, b in zip(single.get_accumulators(), many.get_accumulators()):
        assert rel_l2(b, a) < 1e-6  # the FP32 sum over shots in another order


@pytest.mark.parametrize("nshot,group,nsteps,ntz,ntx", [(1, 1, 3, 1, 1), (5, 2, 4, 2, 3), (4, 4, 5, 1, 4), (7, 3, 2, 3, 1)])
def test_ticket_order_serves_dependencies_first(nshot, group, nsteps, ntz, ntx):
    """Every item is ticketed once, and after all items it waits for: its own
    column and the four beside it, one step earlier (the order of item_of in
    csrc/stencil.cuh).  With that, the waits of the time loops end for any
    number of resident CTAs."""
    ncol = ntz * ntx

    def item(ticket):
        first = ticket // (nsteps * ncol * group) * group
        r = ticket % (nsteps * ncol * group)
        per_step = min(group, nshot - first) * ncol
        t, q = divmod(r, per_step)
        return first + q // ncol, t, q % ncol

    seen = {}
    for k in range(nshot * nsteps * ncol):
        s, t, c = item(k)
        assert 0 <= s < nshot and 0 <= t < nsteps and (s, t, c) not in seen
        if t:
            z, x = c % ntz, c // ntz
            beside = [(z, x), (z - 1, x), (z + 1, x), (z, x - 1), (z, x + 1)]
            for zz, xx in beside:
                if 0 <= zz < ntz and 0 <= xx < ntx:
                    assert seen[s, t - 1, zz + ntz * xx] < k
        seen[s, t, c] = k
    assert len(seen) == nshot * nsteps * ncol
