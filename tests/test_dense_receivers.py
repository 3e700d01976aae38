"""Receivers in every cell of a volume with a long y axis: sampling that falls
behind the time loop must not see a later step, whatever the tile."""
import numpy as np
import pytest

import oracle as orc
from cases import TOL_IMAGE, TOL_SEIS, context, indices, oracle_wavelet, rel_l2
from fwi3d_b200 import lib, synth

NZ, NX, NY, NB, DH, NT = 12, 10, 208, 4, 10.0, 260


def _workload(nsrc=1):
    """4400 m/s and a source in the middle, so that the wave reaches both ends
    of the y axis; 300 receivers more on one cell."""
    rng = np.random.default_rng(5)
    v = (4000 + 400 * rng.random((NY, NX, NZ))).astype(np.float32)
    k, j, i = np.meshgrid(np.arange(NY), np.arange(NX), np.arange(NZ), indexing="ij")
    rec = np.stack([j.ravel() * DH, k.ravel() * DH, i.ravel() * DH], 1).astype(np.float32)
    rec = np.concatenate([rec, np.repeat(rec[100 * NX * NZ:100 * NX * NZ + 1], 300, 0)])
    src = np.array([[40.0, 1040.0 + 40.0 * s, 50.0] for s in range(nsrc)], np.float32)
    return synth.Workload("dense", NZ, NX, NY, DH, NT, 1e-3, 60.0, NB, v, src, rec, abc_factor=0.01)


def _line(i, j):
    """Receivers of one (z, x) line, one per y plane."""
    return np.arange(NY) * (NX * NZ) + j * NZ + i


@pytest.mark.gpu
@pytest.mark.parametrize("boundary", [lib.BOUNDARY_ABC, lib.BOUNDARY_RBC])
def test_dense_samples_equal_sparse_ones_on_every_tile(boundary):
    w = _workload()
    dense = context(w, boundary)
    dense.set_velocity(w.vp)
    lines = [_line(i, j) for i, j in ((0, 0), (5, 4), (11, 9), (3, 7))]
    sparse = []
    for at in lines:
        c = context(synth.Workload("line", NZ, NX, NY, DH, NT, 1e-3, 60.0, NB, w.vp, w.src, w.rec[at],
                                   abc_factor=w.abc_factor), boundary)
        c.set_velocity(w.vp)
        sparse.append(c)
    src, rec = indices(w, NB)
    w64, _ = oracle_wavelet(dense, w)
    ref = orc.forward(dense.get_padded_velocity(), DH, w.dt, NT, dense.tlag, w64, src[0], rec,
                      abc=boundary == lib.BOUNDARY_ABC, nb=NB, factor=w.abc_factor)[0]
    assert np.abs(ref[[0, NY * NX * NZ - 1], -60:]).max() > 0.0
    for tile in range(-1, len(lib.tile_table())):
        dense.set_tiles(tile, -1)
        first = dense.model_shots([0])[0]
        assert rel_l2(first, ref) < TOL_SEIS, tile
        assert np.array_equal(first[NY * NX * NZ:], np.repeat(first[100 * NX * NZ:100 * NX * NZ + 1], 300, 0))
        for c, at in zip(sparse, lines):
            c.set_tiles(tile, -1)
            assert np.array_equal(c.model_shots([0])[0], first[at]), tile
        for _ in range(3):
            assert np.array_equal(dense.model_shots([0])[0], first), tile


@pytest.mark.gpu
def test_dense_samples_of_shots_side_by_side():
    w = _workload(nsrc=5)
    single, many = context(w, lib.BOUNDARY_RBC), context(w, lib.BOUNDARY_RBC, max_batch=4)
    for c in (single, many):
        c.set_velocity(w.vp)
    ids = list(range(5))
    for a, b in zip(single.model_shots(ids), many.model_shots(ids)):
        assert np.array_equal(a, b)


@pytest.mark.gpu
@pytest.mark.parametrize("boundary", [lib.BOUNDARY_ABC, lib.BOUNDARY_RBC])
def test_a_wall_of_receivers_beside_sparse_columns(boundary):
    """The publishers of a few columns are items behind their compute warps when
    the tickets end; what they still have ahead is published and sampled."""
    n, nb, nt = 121, 20, 60
    v = np.full((n, n, n), 4000.0, np.float32)
    k, i = np.meshgrid(np.arange(n), np.arange(n), indexing="ij")
    wall = np.stack([np.full(n * n, 60), k.ravel(), i.ravel()], 1) * DH
    k, j = np.meshgrid(np.arange(n), np.arange(0, n, 5), indexing="ij")
    layer = np.stack([j.ravel(), k.ravel(), np.full(j.size, 100)], 1) * DH
    rec = np.concatenate([wall, layer]).astype(np.float32)
    src = np.array([[600.0, 600.0, 900.0]], np.float32)

    def ctx(r):
        w = synth.Workload("wall", n, n, n, DH, nt, 1e-3, 60.0, nb, v, src, r, abc_factor=0.01)
        c = context(w, boundary)
        c.set_velocity(v)
        return c

    parts = [np.arange(n * n)[p::24] for p in range(24)] + [np.arange(n * n, len(rec))]
    dense, sparse = ctx(rec), [ctx(rec[p]) for p in parts]
    for tile in range(-1, len(lib.tile_table())):
        dense.set_tiles(tile, -1)
        got = dense.model_shots([0])[0]
        for c, p in zip(sparse, parts):
            c.set_tiles(tile, -1)
            assert np.array_equal(c.model_shots([0])[0], got[p]), tile
    assert np.abs(got[:, -1]).max() > 0.0


@pytest.mark.gpu
def test_back_propagation_of_a_wall_of_receivers():
    """Adjoint sources on every cell of a wall: linear in the data, so the image
    is the sum of the images of its parts."""
    n, nb, nt = 101, 10, 60
    v = np.full((n, n, n), 4000.0, np.float32)
    k, i = np.meshgrid(np.arange(n), np.arange(n), indexing="ij")
    rec = (np.stack([np.full(n * n, 50), k.ravel(), i.ravel()], 1) * DH).astype(np.float32)
    w = synth.Workload("wall", n, n, n, DH, nt, 1e-3, 60.0, nb, v, np.array([[500.0, 500.0, 700.0]], np.float32), rec)
    data = np.random.default_rng(0).standard_normal((n * n, nt)).astype(np.float32)
    c = context(w, lib.BOUNDARY_RBC)
    c.set_velocity(v)
    for tile in range(-1, len(lib.tile_table())):
        c.set_tiles(-1, tile)
        images = []
        for parts in (1, 16):
            c.reset_accumulators()
            for p in range(parts):
                d = np.zeros_like(data)
                d[p::parts] = data[p::parts]
                c.rtm_shots([0], d)
            images.append(c.get_accumulators()[0])
        assert np.abs(images[0]).max() > 0.0
        assert rel_l2(*images) < TOL_IMAGE, tile
