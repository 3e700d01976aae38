"""The rules of the time-loop kernels (csrc/loop_order.h), compiled for the host:
which items are taken first, what they wait for, and when planes are published."""
import ctypes as C
import random
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "fwi3d_b200" / "csrc"

WRAPPER = """
#include "loop_order.h"
extern "C" {
void item(long long ticket, int nshot, int group, int nsteps, int ncol, int *out)
{
    const fwi::Item it = fwi::item_of(ticket, nshot, group, nsteps, ncol);
    out[0] = it.shot, out[1] = it.t, out[2] = it.col;
}
int dependency(int lane, int col, int ntz, int ncol) { return fwi::dependency_column(lane, col, ntz, ncol); }
int awaited(int p, int nyy) { return fwi::planes_awaited(p, nyy); }
int lead() { return fwi::kSampleLead; }
int next(int published, int stored, int lead) { return fwi::next_publication(published, stored, lead); }
int first(int next, int last, int lead) { return fwi::work_first(next, last, lead); }
}
"""


@pytest.fixture(scope="module")
def rules(tmp_path_factory):
    d = tmp_path_factory.mktemp("loop_order")
    (d / "w.cpp").write_text(WRAPPER)
    subprocess.run(["g++", "-O1", "-std=c++17", "-fPIC", "-shared", f"-I{CSRC}", "-o", d / "w.so", d / "w.cpp"], check=True)
    lib = C.CDLL(str(d / "w.so"))
    lib.item.argtypes = [C.c_longlong, C.c_int, C.c_int, C.c_int, C.c_int, C.POINTER(C.c_int)]
    return lib


def _storable(rules, published, nyy):
    """Planes below this number can be stored by a step whose predecessor has
    published so many."""
    p = 4
    while p < nyy and rules.awaited(p, nyy) <= published:
        p += 1
    return p - 4


def _too_early(rules, nyy, lead, rng):
    """Publishes one item after random stores; a plane that step t+2 may
    overwrite before step t has sampled it, or None."""
    last = nyy - 4
    published = stored = sampled = 4
    while published < last:
        if stored == published:
            stored = min(last, stored + (1 if rng.random() < 0.5 else rng.randint(1, nyy)))
        published = rules.next(published, stored, lead)
        if rules.first(published, last, lead):
            sampled = published
        overwritten = _storable(rules, _storable(rules, published, nyy), nyy)
        if overwritten > sampled:
            return sampled
        sampled = published
    return None


@pytest.mark.parametrize("nyy", [9, 12, 13, 16, 17, 21, 24, 25, 26, 60, 301])
def test_planes_are_sampled_before_they_can_be_overwritten(rules, nyy):
    rng = random.Random(nyy)
    for _ in range(200):
        assert _too_early(rules, nyy, rules.lead(), rng) is None
        assert _too_early(rules, nyy, 0, rng) is None
    # one more plane of lead would be too much where an item is long enough
    if nyy > 2 * rules.lead() + 10:
        assert any(_too_early(rules, nyy, rules.lead() + 1, rng) is not None for _ in range(200))


@pytest.mark.parametrize("nshot,group,nsteps,ntz,ntx", [(1, 1, 3, 1, 1), (5, 2, 4, 2, 3), (4, 4, 5, 1, 4), (7, 3, 2, 3, 1),
                                                        (64, 9, 3, 2, 2)])
def test_items_are_taken_after_all_that_they_wait_for(rules, nshot, group, nsteps, ntz, ntx):
    ncol = ntz * ntx
    taken, it = {}, (C.c_int * 3)()
    for ticket in range(nshot * nsteps * ncol):
        rules.item(ticket, nshot, group, nsteps, ncol, it)
        s, t, c = it
        assert 0 <= s < nshot and 0 <= t < nsteps and 0 <= c < ncol and (s, t, c) not in taken
        z, x = c % ntz, c // ntz
        want = {zz + ntz * xx for zz, xx in ((z, x), (z - 1, x), (z + 1, x), (z, x - 1), (z, x + 1))
                if 0 <= zz < ntz and 0 <= xx < ntx}
        waits = [rules.dependency(lane, c, ntz, ncol) for lane in range(32)]
        assert sorted(w for w in waits if w >= 0) == sorted(want) and waits[0] == c
        if t:
            assert all(taken[s, t - 1, w] < ticket for w in want)
        taken[s, t, c] = ticket
    assert len(taken) == nshot * nsteps * ncol


def test_tickets_beyond_32_bits(rules):
    nshot, group, nsteps, ncol = 61, 4, 200_003, 1_003  # 12.2e9 items, a last group of one shot
    it = (C.c_int * 3)()
    for s, t, c in ((0, 0, 0), (3, nsteps - 1, ncol - 1), (8, 5, 7), (59, nsteps - 1, 1), (60, 0, 0), (60, nsteps - 1, 1_002)):
        first = s // group * group
        per_step = min(group, nshot - first) * ncol
        ticket = first * nsteps * ncol + t * per_step + (s - first) * ncol + c
        rules.item(ticket, nshot, group, nsteps, ncol, it)
        assert tuple(it) == (s, t, c)
