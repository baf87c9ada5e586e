"""One call of many updates against as many calls of one: within a call the
state may be packed, small systems fill their cell lists without a launch of
their own, and the blocks follow the system's size, none of which may change
a bit."""
import numpy as np
import pytest

import nwgb
from nwgb import abi
from nwgb.batch import Batch
from nwgb.init import initial_state, wca_config

pytestmark = pytest.mark.gpu

STATE = (abi.NW_POSITION, abi.NW_VELOCITY, abi.NW_FORCE, abi.NW_FORCE_OLD, abi.NW_TANGENT)


def _planar(nf, L, box, **kw):
    srd = kw.pop("srd", False)
    c = wca_config(nf, L, box, srd=srd, seed=6)
    for k, v in kw.items():
        if k == "walls":
            c.boundary[1] = v
        else:
            setattr(c, k, v)
    return c


def _three(nf, L, grid, **kw):
    c = abi.default_config(abi.NW_MODEL_WCA_WORMS, nf, L, grid, False)
    c.seed = 6
    for k, v in kw.items():
        setattr(c, k, v)
    return c


CASES = {
    "planar": lambda: _planar(60, 10, (60.0, 30.0)),
    "planar_srd": lambda: _planar(60, 10, (60.0, 30.0), srd=True, srd_gap=4),
    "planar_srd_langevin": lambda: _planar(31, 7, (40.0, 30.0), srd=True, srd_gap=3, langevin_with_srd=1),
    "channel": lambda: _planar(40, 9, (50.0, 40.0), walls=abi.NW_WALL),
    "channel_no_slip": lambda: _planar(40, 9, (50.0, 40.0), walls=abi.NW_WALL_NO_SLIP),
    "eager_tangents": lambda: _planar(90, 3, (40.0, 30.0)),
    "one_bead": lambda: _planar(50, 1, (30.0, 30.0)),
    "longest_packed": lambda: _planar(4, 256, (230.0, 12.0)),
    "too_long_to_pack": lambda: _planar(4, 257, (230.0, 12.0)),
    "reversal": lambda: _planar(60, 10, (60.0, 30.0), reverse_probability=0.2),
    "sixteen_slots": lambda: _planar(60, 10, (60.0, 30.0), cell_capacity=16),
    "short_lists": lambda: _planar(60, 10, (60.0, 30.0), neighbor_skin=0.05),
    "largest_inserting": lambda: _planar(8192, 16, (520.0, 420.0)),
    "first_not_inserting": lambda: _planar(8193, 16, (520.0, 420.0)),
    "three_d": lambda: _three(40, 8, (9, 10, 11)),
    "three_d_large": lambda: _three(6000, 13, (48, 49, 50)),
    "cell_lists": lambda: _planar(60, 10, (60.0, 30.0), strategy=abi.NW_STRATEGY_CELL_LISTS),
}


def _state(c):
    if c.dim == 2:
        pos, vel = initial_state(c, seed=2, layout="rows")
        pos[: c.n_beads, 2] = np.linspace(-0.2, 0.2, c.n_beads)  # z and radius are carried
        pos[: c.n_beads, 3] = np.linspace(0.4, 0.6, c.n_beads)
        vel[: c.n_beads, 2] = np.linspace(-0.1, 0.1, c.n_beads)
        return pos, vel
    rng = np.random.default_rng(3)
    nb, L = c.n_beads, c.filament_size
    box = np.array([c.box[a] for a in range(3)])
    pos, vel = np.zeros((nb, 4), np.float32), np.zeros((nb, 4), np.float32)
    per, ny = int(box[0] // (L * 0.8 + 1.0)), int(box[1] // 1.2)
    w = np.arange(c.num_filaments)
    x = (w % per)[:, None] * (box[0] / per) + np.arange(L) * 0.8
    y, z = ((w // per) % ny + 0.5) * (box[1] / ny), (w // (per * ny) + 0.5) * 1.2
    pos[:, :3] = np.stack([x, *np.broadcast_arrays(y[:, None], z[:, None] + 0 * x)], -1).reshape(-1, 3)
    pos[:, :3] = np.array([c.origin[a] for a in range(3)]) + np.mod(pos[:, :3], box)
    vel[:, :3] = rng.normal(0, 0.3, (nb, 3))
    pos[:, 3], vel[:, 3] = c.radius, c.mass
    return pos, vel


@pytest.mark.parametrize("name", sorted(CASES))
def test_one_call_equals_single_updates(name):
    c = CASES[name]()
    c.kT = c.srd_kT = 0.4  # list builds within the run
    pos, vel = _state(c)
    out = []
    for calls in ([24], [1] * 24, [2, 5, 1, 9, 7], [3, 21]):
        with nwgb.System(c) as s:
            s.set_array(abi.NW_POSITION, pos)
            s.set_array(abi.NW_VELOCITY, vel)
            for n in calls:
                s.step(n)
            s.sync()
            out.append([s.get_array(a) for a in STATE])
    for other in out[1:]:
        for which, x, y in zip(STATE, out[0], other):
            assert np.array_equal(x.view(np.uint32), y.view(np.uint32)), which


def test_batch_call_equals_single_updates():
    """The batch's packed calls and its list kernel over replicas of one block
    and of many."""
    cfgs = [_planar(nf, L, box, activity=0.2 * k) for k, (nf, L, box) in
            enumerate([(3, 5, (20.0, 20.0)), (900, 11, (150.0, 100.0)), (60, 30, (90.0, 40.0)), (1, 7, (15.0, 15.0))])]
    out = []
    for calls in ([20], [1] * 20, [2, 7, 11]):
        with Batch(cfgs) as b:
            for r, c in enumerate(cfgs):
                pos, vel = _state(c)
                b.set_array(r, abi.NW_POSITION, pos)
                b.set_array(r, abi.NW_VELOCITY, vel)
            for n in calls:
                b.step(n)
            b.sync()
            out.append([b.get_array(r, a) for r in range(len(cfgs)) for a in STATE])
    for other in out[1:]:
        for x, y in zip(out[0], other):
            assert np.array_equal(x.view(np.uint32), y.view(np.uint32))
