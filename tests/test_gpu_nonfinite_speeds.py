"""Temperatures of states with velocities or masses that are not numbers: they
are those of double-precision sums, not those of the other particles."""
import numpy as np
import pytest

import nwgb
from nwgb import abi
from nwgb.init import initial_state, wca_config

import observables_oracle as obs

pytestmark = pytest.mark.gpu

NAN, INF = float("nan"), float("inf")


def _observe(cfg, pos, vel):
    with nwgb.System(cfg) as s:
        s.set_array(abi.NW_POSITION, pos)
        s.set_array(abi.NW_VELOCITY, vel)
        return s.observe()


def _check(got, vel, nb, dim):
    for k, v in (("bead_temperature", vel[:nb]), ("solvent_temperature", vel[nb:])):
        with np.errstate(invalid="ignore"):
            want = obs.temperature(v, dim)
        if np.isfinite(want):
            assert abs(got[k] - want) <= 1e-12 * want, k
        else:
            assert np.array_equal(got[k], want, equal_nan=True), (k, got[k], want)


@pytest.mark.parametrize("speed", [(NAN, NAN), (NAN, 0.0), (0.0, NAN), (NAN, 0.3), (INF, 0.0), (INF, NAN), (-INF, 1.0)])
@pytest.mark.parametrize("where", ["bead", "solvent"])
def test_planar(speed, where):
    cfg = wca_config(40, 7, (37.0, 29.0), srd=True, seed=2)
    pos, vel = initial_state(cfg, seed=2, layout="rows")
    vel[17 if where == "bead" else cfg.n_beads + 1234, :2] = speed
    _check(_observe(cfg, pos, vel), vel, cfg.n_beads, 2)


@pytest.mark.parametrize("speed", [(NAN, 0.0, 0.0), (0.0, 0.0, NAN), (NAN, NAN, NAN), (0.1, NAN, 0.2), (0.0, INF, 0.0)])
def test_three_dimensions(speed):
    cfg = abi.default_config(abi.NW_MODEL_WCA_WORMS, 20, 5, (9, 10, 11), False)
    rng = np.random.default_rng(1)
    pos, vel = np.zeros((100, 4), np.float32), np.zeros((100, 4), np.float32)
    pos[:, :3], vel[:, :3], vel[:, 3] = rng.uniform(0, 9, (100, 3)), rng.normal(0, 0.3, (100, 3)), 1.0
    vel[63, :3] = speed
    _check(_observe(cfg, pos, vel), vel, 100, 3)
