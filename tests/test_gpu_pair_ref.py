"""The REF_DEM pair pass from the sorted runs at grid edges: narrow and
aliased grids, crowded and empty cells against the oracle; odd modulo grids,
which the oracle's REF_DEM (masks, as the reference) does not have, against
the cell-list strategy's own pair kernel."""
import numpy as np
import pytest

import nwgb
from nwgb import abi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("grid,hash_mode", [
    ((4, 4), abi.NW_HASH_MASK), ((8, 2), abi.NW_HASH_MASK), ((2, 8), abi.NW_HASH_MASK), ((1, 16), abi.NW_HASH_MASK),
    ((32, 4), abi.NW_HASH_MASK), ((5, 7), abi.NW_HASH_MODULO), ((3, 3), abi.NW_HASH_MODULO), ((33, 6), abi.NW_HASH_MODULO),
])
@pytest.mark.parametrize("density", [0.3, 2.5])
def test_forces_at_grid_edges(orc, grid, hash_mode, density):
    L = 5
    nf = max(1, int(density * grid[0] * grid[1] / L))
    c = abi.default_config(abi.NW_MODEL_REF_DEM, nf, L, (8, 8, 1), False)
    c.grid[0], c.grid[1], c.hash_mode = grid[0], grid[1], hash_mode
    c.bond_r0, c.activity, c.seed = 0.8, 0.5, 4
    abi.check(nwgb.load_library().nw_config_finalize(abi.C.byref(c)))
    rng = np.random.default_rng(grid[0] * 100 + grid[1])
    nb = c.n_beads
    pos, vel = np.zeros((nb, 4), np.float32), np.zeros((nb, 4), np.float32)
    box = np.array([c.box[0], c.box[1]])
    a = rng.uniform(0, 2 * np.pi, (nf, 1))
    k = np.arange(L) * 0.8
    xy = rng.random((nf, 1, 2)) * box + np.stack([k * np.cos(a), k * np.sin(a)], -1)
    pos[:, :2] = np.array([c.origin[0], c.origin[1]]) + np.mod(xy.reshape(-1, 2), box)
    pos[:, 3], vel[:, 3] = c.radius, c.mass
    vel[:, :2] = rng.normal(0, 0.3, (nb, 2))
    zeros = np.zeros((nb, 4), np.float32)
    with nwgb.System(c) as s:
        s.set_array(abi.NW_POSITION, pos)
        s.set_array(abi.NW_VELOCITY, vel)
        s.step(1)
        s.sync()
        got = s.get_array(abi.NW_FORCE)
    if hash_mode == abi.NW_HASH_MODULO:
        c.strategy = abi.NW_STRATEGY_CELL_LISTS
        c.cell_capacity = 16
        with nwgb.System(c) as s:
            s.set_array(abi.NW_POSITION, pos)
            s.set_array(abi.NW_VELOCITY, vel)
            s.step(1)
            s.sync()
            want = s.get_array(abi.NW_FORCE)
        # the same terms summed in another order: rounding of the largest sums
        assert np.abs(got - want).max() < 1e-5 * np.abs(want).max()
        return
    st = dict(pos=pos, vel=vel, force=zeros, force_old=zeros, tangent=zeros)
    ref = orc.step(c, st, 0, c.dt, prec=32)["force"]
    scale = orc.step(c, st, 0, c.dt, prec=64, force_scale=True)["force_scale"]
    err = np.linalg.norm(got[:, :3].astype(np.float64) - ref[:, :3], axis=1) / scale
    assert float(err.max()) < 1e-5  # the bar of every one-step force
