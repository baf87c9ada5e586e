"""Beads set several boxes away are wrapped by one box per update; until they
are inside, their forces on beads well inside the box are those of the images,
as the cell-list strategy, which knows no list from an earlier update, takes
them."""
import numpy as np
import pytest

import nwgb
from nwgb import abi
from nwgb.batch import Batch
from nwgb.init import wca_config

pytestmark = pytest.mark.gpu

# Rows 1.0 apart, every other row two to four boxes away: the forces that cross
# rows are 24 epsilon a bead.  The strategies sum the same pairs in another
# order, so a position differs by at most the odd flip of its last bit, 8e-6 at
# 128, times the pairs' stiffness, about 700: 0.006 a flip.
TOL = 0.05
FAR = ((3, 0, 0), (0, -2, 0), (-2, 3, 0), (4, 0, 0))


def _rows(c, layers):
    L, nf = c.filament_size, c.num_filaments
    pos, vel = np.zeros((nf, L, 4), np.float32), np.zeros((nf * L, 4), np.float32)
    for w in range(nf):
        # filaments of the first half stay inside, those of the second are far
        far, k = divmod(w, nf // 2)
        row, rest = 2 * (k % 8) + far, k // 8
        pos[w, :, 0] = c.origin[0] + 4.0 + 10.0 * (rest % 2) + 0.8 * np.arange(L)
        pos[w, :, 1] = c.origin[1] + 4.0 + row
        pos[w, :, 2] = c.origin[2] + 4.0 + 3.0 * (rest // 2) if layers > 1 else 0.0
        if far:
            pos[w, :, :3] += np.array(FAR[k % 4]) * [c.box[a] for a in range(3)]
            if layers > 1:
                pos[w, :, 2] += (k % 3 - 1) * 2 * c.box[2]
    pos[..., 3], vel[:, 3] = c.radius, 1.0
    return pos.reshape(-1, 4), vel


def _config(three):
    if three:
        c = abi.default_config(abi.NW_MODEL_WCA_WORMS, 64, 8, (22, 22, 22), False)
    else:
        c = wca_config(32, 8, (24.0, 24.0))
    c.kT, c.seed = 0.0, 1
    return c


def _forces(c, strategy, calls, pos, vel):
    c.strategy = strategy
    out = []
    with nwgb.System(c) as s:
        s.set_array(abi.NW_POSITION, pos)
        s.set_array(abi.NW_VELOCITY, vel)
        for n in calls:
            s.step(n)
            out.append((s.get_array(abi.NW_FORCE), s.get_array(abi.NW_POSITION)))
        s.sync()
    return out


@pytest.mark.parametrize("three", [False, True])
@pytest.mark.parametrize("calls", [(1, 1, 1, 1, 1, 1), (2, 1, 3), (3, 3)])
def test_forces_of_far_beads(three, calls):
    c = _config(three)
    pos, vel = _rows(c, 3 if three else 1)
    want = _forces(c, abi.NW_STRATEGY_CELL_LISTS, calls, pos, vel)
    got = _forces(c, abi.NW_STRATEGY_VERLET, calls, pos, vel)
    for (fa, pa), (fb, pb) in zip(want, got):
        assert np.abs(fa).max() > 5.0  # pairs do act
        assert np.abs(pa[:, :3] - pb[:, :3]).max() < 1e-4
        assert np.abs(fa[:, :3] - fb[:, :3]).max() < TOL


def test_beads_set_far_during_a_run():
    """Far beads between two calls, through the list's displacement bound."""
    c = _config(False)
    pos, vel = _rows(c, 1)
    inside = pos.copy()
    org = np.array([c.origin[0], c.origin[1]])
    inside[:, :2] = org + np.mod(pos[:, :2] - org, 24.0)
    out = []
    for strategy in (abi.NW_STRATEGY_CELL_LISTS, abi.NW_STRATEGY_VERLET):
        c.strategy = strategy
        with nwgb.System(c) as s:
            s.set_array(abi.NW_POSITION, inside)
            s.set_array(abi.NW_VELOCITY, vel)
            s.step(3)
            p = s.get_array(abi.NW_POSITION)
            s.set_array(abi.NW_POSITION, p + (pos - inside))
            s.step(2)
            out.append(s.get_array(abi.NW_FORCE))
    assert np.abs(out[0][:, :3] - out[1][:, :3]).max() < TOL


@pytest.mark.parametrize("calls", [(2,), (1, 1), (6,)])
def test_batch_of_far_beads(calls):
    c = _config(False)
    pos, vel = _rows(c, 1)
    want = _forces(c, abi.NW_STRATEGY_CELL_LISTS, calls, pos, vel)[-1][0]
    with Batch([_config(False), _config(False)]) as b:
        for r in range(2):
            b.set_array(r, abi.NW_POSITION, pos)
            b.set_array(r, abi.NW_VELOCITY, vel)
        for n in calls:
            b.step(n)
        b.sync()
        for r in range(2):
            got = b.get_array(r, abi.NW_FORCE)
            # noise is off and the replicas' seeds draw nothing else
            assert np.abs(got[:, :3] - want[:, :3]).max() < TOL
