"""Images, illumination and the adjoint field below 2^-126, where FP32 has fewer
digits but does not end: what is added there has to arrive."""
import numpy as np
import pytest

from cases import context, interior, rel_l2
from fwi3d_b200 import lib, synth

pytestmark = pytest.mark.gpu

NT = 70


def _workload(k=0):
    """The same experiment with lengths and times 2^k times as long: FP32 runs
    through the same digits, the source and the adjoint source 2^(-3k) times as
    strong."""
    nz, nx, ny, nb, s = 37, 26, 24, 6, 2.0 ** k
    rng = np.random.default_rng(4)
    v = (1800 + 600 * rng.random((ny, nx, nz))).astype(np.float32)
    x, y = np.arange(nx) * 10.0, np.arange(ny) * 10.0
    rec = synth.surface_grid(x, y, 20.0).astype(np.float32)
    src = np.array([[120.0, 110.0, 200.0]], np.float32)
    return synth.Workload("small", nz, nx, ny, 10.0 * s, NT, 1e-3 * s, 60.0 / s, nb, v, src * np.float32(s),
                          rec * np.float32(s))


def _data(w):
    return np.random.default_rng(1).standard_normal((len(w.rec), NT)).astype(np.float32)


def _context(w, grad):
    c = context(w, lib.BOUNDARY_RBC, flags=lib.FLAG_SUBTRACT_SOURCE | lib.FLAG_GRAD_DY if grad else 0)
    c.set_velocity(w.vp)
    return c


def _run(c, data, grad):
    c.reset_accumulators()
    (c.gradient_shots if grad else c.rtm_shots)([0], data)
    return c.get_accumulators()


@pytest.mark.parametrize("grad", [False, True])
def test_accumulators_keep_what_is_below_the_normal_range(grad):
    w = _workload()
    data, base = _data(w), _context(w, grad)
    img, ill = (a.astype(np.float64) for a in _run(base, data, grad))
    # the image scales as 2^(-6k), the gradient, which has 1/dt, as 2^(-7k);
    # k puts the peak of one accumulator at 2^-130 .. 2^-126
    for which, (ref, power) in enumerate(((img, 7 if grad else 6), (ill, 6))):
        k = int(np.ceil((np.log2(np.abs(ref).max()) + 127) / power))
        scaled = _workload(k)
        c = _context(scaled, grad)
        assert c.tlag == base.tlag
        steps = c.tlag + NT
        want = ref * 2.0 ** (-power * k)
        assert 2.0 ** -135 < np.abs(want).max() < 2.0 ** -126
        for tile in range(-1, len(lib.tile_table())):
            c.set_tiles(-1, tile)
            got = _run(c, data, grad)[which].astype(np.float64)
            # per step a product rounded to a multiple of 2^-149 (the gradient's
            # after two more), and the roundings of the sum at full digits
            assert np.abs(got - want).max() <= 2 * steps * 2.0 ** -149, tile
            assert np.count_nonzero(interior(got, w.nb)) > 0


@pytest.mark.parametrize("grad", [False, True])
def test_what_is_not_added_to_keeps_its_bits(grad):
    """No data, so no adjoint field: the image keeps every value, and the
    illumination those outside the physical box."""
    import torch
    w = _workload()
    c = _context(w, grad)
    rng = np.random.default_rng(9)
    shape = c.padded_shape
    preset = (rng.standard_normal(shape) * 2.0 ** rng.integers(-150, -100, shape)).astype(np.float32)
    assert np.count_nonzero((preset != 0) & (np.abs(preset) < 2.0 ** -126)) > 1000
    d = torch.from_numpy(preset).cuda()
    torch.cuda.synchronize()
    inside = np.zeros(shape, bool)
    inside[w.nb:-w.nb, w.nb:-w.nb, w.nb:-w.nb] = True
    for tile in range(-1, len(lib.tile_table())):
        c.set_tiles(-1, tile)
        c.set_accumulators_dev(d.data_ptr(), d.data_ptr())
        (c.gradient_shots if grad else c.rtm_shots)([0], np.zeros((len(w.rec), NT), np.float32))
        img, ill = c.get_accumulators()
        assert np.array_equal(img, preset), tile
        assert np.array_equal(ill[~inside], preset[~inside]), tile
        assert (ill[inside] > 0).any()


def test_adjoint_sources_below_the_normal_range():
    w = _workload()
    data, c = _data(w), _context(w, False)
    img = _run(c, data, False)[0].astype(np.float64)
    # idh3 * data at 2^-127 and below; the field rounds to multiples of 2^-149
    # each step, three times, which the wave equation adds up over at most N^2 / 2
    # steps: 3 * 130^2 / 2 * 2^-150 = 2^-135.4 of about 2^-128
    m = int(np.ceil(np.log2(np.abs(data).max() * 1e-3) + 127))
    assert m > 100
    tiny = (data * np.float32(2.0 ** -60)) * np.float32(2.0 ** (60 - m))
    assert np.abs(tiny).max() > 0
    for tile in range(-1, len(lib.tile_table())):
        c.set_tiles(-1, tile)
        got = _run(c, tiny, False)[0].astype(np.float64)
        assert rel_l2(got * 2.0 ** m, img) < 2e-2, tile


@pytest.mark.parametrize("grad", [False, True])
def test_sums_beyond_the_scaled_range(grad):
    """Data so large that the image times 2^24 is no FP32 number: it comes from the
    loop that sums without a scale, and the illumination is counted once."""
    w = _workload()
    data, c = _data(w), _context(w, grad)
    img, ill = (a.astype(np.float64) for a in _run(c, data, grad))
    m = int(np.floor(125 - np.log2(np.abs(img).max())))
    big = (data * np.float32(2.0 ** 60)) * np.float32(2.0 ** (m - 60))
    assert np.isfinite(big).all() and np.abs(img).max() * 2.0 ** (m + 24) > np.finfo(np.float32).max
    for tile in (-1, 0, 6):
        c.set_tiles(-1, tile)
        c.reset_accumulators()
        for _ in range(2):  # and once more on top
            (c.gradient_shots if grad else c.rtm_shots)([0], big)
        got = c.get_accumulators()
        # the same FP32 products, summed in another order over 2 x 130 steps
        assert rel_l2(got[0].astype(np.float64) * 2.0 ** -m, 2 * img) < 1e-5, tile
        assert rel_l2(got[1], 2 * ill) < 1e-5, tile


def test_cells_of_half_a_millimetre():
    """Fields 2^42 times as strong, whose illumination times 2^24 could leave the
    range: summed without a scale from the start."""
    w = _workload()
    data = _data(w)
    img, ill = (a.astype(np.float64) for a in _run(_context(w, False), data, False))
    c = _context(_workload(-14), False)
    for tile in range(-1, len(lib.tile_table())):
        c.set_tiles(-1, tile)
        got = _run(c, data, False)
        for a, b in zip(got, (img, ill)):
            assert rel_l2(a * 2.0 ** -84, b) < 1e-5, tile
