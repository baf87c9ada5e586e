"""SRD collisions that find their members through the solvent's stored cell
order against collisions that bucket the solvent (the path taken after the
solvent's positions were written from outside): the same members in the same
order, so the same bits."""
import numpy as np
import pytest

import nwgb
from nwgb import abi
from nwgb.init import initial_state, wca_config

pytestmark = pytest.mark.gpu

ARRAYS = (abi.NW_POSITION, abi.NW_VELOCITY, abi.NW_SRD_SORTED_INDEX, abi.NW_SRD_CELL_START, abi.NW_SRD_CELL_END,
          abi.NW_SRD_CELL_MEAN)


def _wca(box, nf=12, L=5, walls=(), kT=0.1, gap=3, density=4.0):
    c = wca_config(nf, L, box, srd=True, srd_density=density, seed=3)
    c.srd_gap, c.srd_kT = gap, kT
    for a in walls:
        c.boundary[a] = abi.NW_WALL
    return c


def _wca3(grid, walls=()):
    c = abi.default_config(abi.NW_MODEL_WCA_WORMS, 6, 4, grid, False)
    c.srd_enabled, c.srd_gap, c.seed, c.srd_alpha, c.num_solvent = 1, 2, 5, 2.26893, 4
    for a in range(3):
        c.srd_grid[a] = int(c.box[a])
        c.srd_cell_size[a] = c.box[a] / c.srd_grid[a]
        c.num_solvent *= c.srd_grid[a]
    for a, kind in walls:
        c.boundary[a] = kind
    return c


def _dem(grid, layers=1):
    c = abi.default_config(abi.NW_MODEL_REF_DEM, 10, 6, (grid, grid, layers), True)
    c.srd_kT, c.seed = 0.1, 9
    return c


CASES = {
    "odd": lambda: _wca((47.0, 31.0)),
    "wide": lambda: _wca((210.0, 17.0), density=3.0),
    "channel": lambda: _wca((40.0, 37.0), walls=(1,)),
    "closed_box": lambda: _wca((33.0, 29.0), walls=(0, 1)),
    "narrow": lambda: _wca((38.0, 7.0), nf=3, L=3),
    "hot": lambda: _wca((41.0, 43.0), kT=400.0, gap=10),  # steps of about a cell
    "very_hot": lambda: _wca((41.0, 43.0), kT=1e5, gap=10),  # beyond the ordered path
    "crowded": lambda: _wca((23.0, 24.0), density=14.0),  # cells above one lane's share
    "three_d": lambda: _wca3((11, 13, 12)),
    "three_d_walls": lambda: _wca3((11, 12, 13), ((0, abi.NW_WALL), (2, abi.NW_WALL_NO_SLIP))),
    "two_layers": lambda: _wca3((12, 12, 3)),
    "mask_hash": lambda: _dem(64),
    "mask_hash_3d": lambda: _dem(16, 8),
    "mask_hash_tiny": lambda: _dem(8),
}


def _state(c):
    rng = np.random.default_rng(1)
    if c.model == abi.NW_MODEL_WCA_WORMS and c.dim == 2:
        return initial_state(c, seed=2, layout="rows")
    nb, n = c.n_beads, c.n_beads + c.n_solvent
    box = np.array([c.box[a] for a in range(3)])
    org = np.array([c.origin[a] for a in range(3)])
    pos, vel = np.zeros((n, 4), np.float32), np.zeros((n, 4), np.float32)
    pos[:, :3] = org + rng.random((n, 3)) * box
    L = c.filament_size
    for w in range(c.num_filaments):  # straight worms along x, well apart
        b = slice(w * L, (w + 1) * L)
        pos[b, 0] = org[0] + np.mod(0.5 + np.arange(L) * c.bond_r0, box[0])
        pos[b, 1] = org[1] + (w % 5 + 0.5) * box[1] / 5
        pos[b, 2] = org[2] + (w // 5 + 0.5) * box[2] / 2
    if c.grid[2] == 1:
        pos[:, 2] = 0.0
    vel[:, :3] = rng.normal(0, 0.3, (n, 3))
    pos[:nb, 3], vel[:nb, 3], vel[nb:, 3] = c.radius, c.mass, c.solvent_mass
    return pos, vel


@pytest.mark.parametrize("name", sorted(CASES))
def test_ordered_collisions_equal_bucketed_ones(name):
    c = CASES[name]()
    pos, vel = _state(c)
    nb = c.n_beads
    out = []
    for rebucket in (False, True):
        with nwgb.System(c) as s:
            s.set_array(abi.NW_POSITION, pos)
            s.set_array(abi.NW_VELOCITY, vel)
            frames = []
            for _ in range(9):
                if rebucket:
                    s.set_array(abi.NW_POSITION, s.get_array(abi.NW_POSITION, nb, c.n_solvent), nb)
                s.step(int(c.srd_gap))
                frames.append([s.get_array(a) for a in ARRAYS])
            flags = s.error_word()
            assert not flags & abi.NW_EFLAG_BAD_INDEX
            out.append(frames)
    for k, (a, b) in enumerate(zip(*out)):
        for which, x, y in zip(ARRAYS, a, b):
            assert np.array_equal(x.view(np.uint32), y.view(np.uint32)), (name, k, which)


def test_collisions_at_given_shifts():
    """nw_srd_collide with shifts far apart (several cells between two grids)."""
    c = _wca((29.0, 31.0))
    pos, vel = _state(c)
    nb = c.n_beads
    shifts = [(0.0, 0.0, 0.0), (0.49, -0.49, 0.0), (-0.5, 0.5, 0.0), (2.3, -3.7, 0.0), (7.0, 7.0, 0.0), (-29.0, 0.1, 0.0)]
    out = []
    for rebucket in (False, True):
        with nwgb.System(c) as s:
            s.set_array(abi.NW_POSITION, pos)
            s.set_array(abi.NW_VELOCITY, vel)
            frames = []
            for sh in shifts:
                if rebucket:
                    s.set_array(abi.NW_POSITION, s.get_array(abi.NW_POSITION, nb, c.n_solvent), nb)
                s.srd_collide(0.05, sh)
                frames.append([s.get_array(a) for a in ARRAYS])
            assert not s.error_word() & abi.NW_EFLAG_BAD_INDEX
            out.append(frames)
    for k, (a, b) in enumerate(zip(*out)):
        for which, x, y in zip(ARRAYS, a, b):
            assert np.array_equal(x.view(np.uint32), y.view(np.uint32)), (k, which)
