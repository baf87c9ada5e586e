"""SRD collisions of boxes and shifts far from the origin, where coordinates
and shifts round by a good part of a cell: the members found through the
solvent's stored cell order are those of the cells' hashes, as when the
solvent is bucketed."""
import numpy as np
import pytest

import nwgb
from nwgb import abi
from nwgb.init import wca_config

pytestmark = pytest.mark.gpu

ARRAYS = (abi.NW_POSITION, abi.NW_VELOCITY, abi.NW_SRD_SORTED_INDEX, abi.NW_SRD_CELL_START, abi.NW_SRD_CELL_END,
          abi.NW_SRD_CELL_MEAN)


def _system(box, origin, walls=(), speed=0.01):
    c = wca_config(4, 5, box, srd=True, seed=3)
    for a in range(2):
        c.origin[a] = origin[a]
    for a in walls:
        c.boundary[a] = abi.NW_WALL
    c.srd_kT = speed * speed
    rng = np.random.default_rng(4)
    nb, n = c.n_beads, c.n_beads + c.n_solvent
    pos, vel = np.zeros((n, 4), np.float32), np.zeros((n, 4), np.float32)
    pos[:, :2] = (np.array(origin) + rng.random((n, 2)) * np.array(box)).astype(np.float32)
    for w in range(4):
        b = slice(w * 5, (w + 1) * 5)
        pos[b, 0] = origin[0] + 2.0 + np.arange(5)
        pos[b, 1] = origin[1] + 2.0 + 4.0 * w
    vel[:, :2] = rng.normal(0, speed, (n, 2))
    pos[:nb, 3], vel[:, 3] = c.radius, 1.0
    return c, pos, vel


def _frames(c, pos, vel, shifts, dt, rebucket):
    nb, out = c.n_beads, []
    with nwgb.System(c) as s:
        s.set_array(abi.NW_POSITION, pos)
        s.set_array(abi.NW_VELOCITY, vel)
        for sh in shifts:
            if rebucket:
                s.set_array(abi.NW_POSITION, s.get_array(abi.NW_POSITION, nb, c.n_solvent), nb)
            s.srd_collide(dt, sh)
            out.append([s.get_array(a) for a in ARRAYS])
        assert not s.error_word() & abi.NW_EFLAG_BAD_INDEX
    return out


def _compare(c, pos, vel, shifts, dt=0.05):
    a, b = (_frames(c, pos, vel, shifts, dt, r) for r in (False, True))
    n = c.n_beads + c.n_solvent
    for k, (x, y) in enumerate(zip(a, b)):
        assert np.array_equal(np.sort(x[2]), np.arange(n)), k  # every particle once
        for which, p, q in zip(ARRAYS, x, y):
            assert np.array_equal(p.view(np.uint32), q.view(np.uint32)), (k, which)


def _shifts(size=0.5, n=12):
    rng = np.random.default_rng(7)
    return [tuple(rng.uniform(-size, size, 2)) + (0.0,) for _ in range(n)]


@pytest.mark.parametrize("origin", [(-3e4, 1e4), (1e5, -1e5), (1e6, 7.0), (0.0, 4e6), (3e7, 3e7)])
@pytest.mark.parametrize("walls", [(), (1,)])
def test_far_boxes(origin, walls):
    """Two shifts that round to none, steps of a fifth of the distance of
    neighbouring coordinates (and up to all of it): those that round to it take
    particles over cell edges against the difference of the shifts."""
    ulp = float(np.spacing(np.float32(max(abs(o) for o in origin))))
    c, pos, vel = _system((100.0, 60.0), origin, walls, speed=4.0 * ulp)
    _compare(c, pos, vel, [((-1) ** k * 0.49 * ulp, (-1) ** k * 0.49 * ulp, 0.0) for k in range(12)])
    _compare(c, pos, vel, _shifts())


@pytest.mark.parametrize("far", [1e3, 2e4, 1e6])
def test_far_shifts(far):
    c, pos, vel = _system((100.0, 60.0), (0.0, 0.0))
    _compare(c, pos, vel, [(x + far, y - far, 0.0) for x, y, _ in _shifts(0.01)])


@pytest.mark.parametrize("origin", [(0.0, 0.0), (-50.0, -30.0), (1e3, 1e3)])
def test_usual_boxes(origin):
    c, pos, vel = _system((100.0, 60.0), origin, speed=0.3)
    _compare(c, pos, vel, _shifts())


@pytest.mark.parametrize("kind", [abi.NW_WALL, abi.NW_WALL_NO_SLIP])
@pytest.mark.parametrize("axes", [(1,), (0, 1)])
def test_solvent_outside_walls(axes, kind):
    """Solvent set some cells outside the walls is put back by a step longer
    than its streaming; with shifts of a few cells that takes it to cells other
    than the one at the wall."""
    c, pos, vel = _system((41.0, 37.0), (0.0, 0.0), axes, speed=0.3)
    for a in axes:
        c.boundary[a] = kind
    rng = np.random.default_rng(5)
    nb = c.n_beads
    out = nb + rng.permutation(c.n_solvent)[: c.n_solvent // 5]
    for a in axes:
        far = rng.uniform(0.5, 3.0, len(out))
        pos[out, a] = np.where(rng.random(len(out)) < 0.5, -far, c.box[a] + far)
    _compare(c, pos, vel, [(2.3, 2.3, 0.0), (2.3, 2.3, 0.0), (2.4, 2.2, 0.0), (-2.3, -2.4, 0.0), (-2.3, -2.4, 0.0)])
