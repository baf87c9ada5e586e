"""Which path the SRD collisions of tests/test_gpu_srd_order.py and
tests/test_gpu_srd_far.py take, so that their comparisons are of two paths."""
import numpy as np
import pytest

import nwgb
from nwgb import abi

import test_gpu_srd_far as far
import test_gpu_srd_order as order

pytestmark = pytest.mark.gpu


# Solvent whose fastest particle moves by more cells than are looked at (4).
BEYOND = ("hot", "very_hot")


def _paths(c, pos, vel, rebucket=False, frames=None):
    """Whether each of nine collisions took the cell order."""
    out, nb = [], c.n_beads
    with nwgb.System(c) as s:
        s.set_array(abi.NW_POSITION, pos)
        s.set_array(abi.NW_VELOCITY, vel)
        for _ in range(9):
            if rebucket:
                s.set_array(abi.NW_POSITION, s.get_array(abi.NW_POSITION, nb, c.n_solvent), nb)
            s.step(int(c.srd_gap))
            out.append(s.srd_ordered)
            if frames is not None:
                frames.append([s.get_array(a) for a in order.ARRAYS])
        assert not s.error_word() & abi.NW_EFLAG_BAD_INDEX
    return out


@pytest.mark.parametrize("name", sorted(order.CASES))
def test_path_of_the_order_cases(name):
    c = order.CASES[name]()
    pos, vel = order._state(c)
    taken = _paths(c, pos, vel)
    assert not taken[0]  # positions from outside
    assert not any(taken) if name in BEYOND else any(taken)
    assert not any(_paths(c, pos, vel, rebucket=True))


@pytest.mark.parametrize("kT", [3.0, 10.0, 20.0])
@pytest.mark.parametrize("walls", [(), (0, 1)])
def test_steps_of_about_a_cell(kT, walls):
    """Fastest particles of a good part of a cell to somewhat over one, in order
    and bucketed: the same bits."""
    c = order._wca((41.0, 43.0), walls=walls, kT=kT, gap=10)
    pos, vel = order._state(c)
    a, b = [], []
    taken = _paths(c, pos, vel, frames=a)
    assert any(taken[1:])
    _paths(c, pos, vel, rebucket=True, frames=b)
    for k, (x, y) in enumerate(zip(a, b)):
        for which, p, q in zip(order.ARRAYS, x, y):
            assert np.array_equal(p.view(np.uint32), q.view(np.uint32)), (k, which)


@pytest.mark.parametrize("origin,ordered", [((0.0, 0.0), True), ((-3e4, 1e4), True), ((1e6, 7.0), True), ((0.0, 4e6), False), ((3e7, 3e7), False)])
def test_path_of_far_boxes(origin, ordered):
    """Rounding of up to a cell widens the search, of several cells ends it."""
    c, pos, vel = far._system((100.0, 60.0), origin, speed=1e-3)
    with nwgb.System(c) as s:
        s.set_array(abi.NW_POSITION, pos)
        s.set_array(abi.NW_VELOCITY, vel)
        for k in range(4):
            s.srd_collide(0.05, (0.1, 0.1, 0.0))
            assert s.srd_ordered == (ordered and k > 0)
