"""Receivers in every cell of a volume with a long y axis: sampling that falls
behind the time loop must not see a later step, whatever the tile."""
import numpy as np
import pytest

import oracle as orc
from cases import TOL_SEIS, context, indices, oracle_wavelet, rel_l2
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
