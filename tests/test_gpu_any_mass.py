"""Temperatures of particles of any mass: those of double-precision sums, also
where a mass is far from one, not a number, or belongs to a resting particle."""
import numpy as np
import pytest

import nwgb
from nwgb import abi
from nwgb.init import initial_state, wca_config

import observables_oracle as obs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mass", [float("nan"), float("inf"), 0.0, 1e-38, 1e-30, 1e-9, 0.01, 900.0, 1e5, 1e20, 3e38, -2.0])
@pytest.mark.parametrize("scale", [0.0, 1e-13, 1.0, 1e13])
@pytest.mark.parametrize("every", [1, 3])
def test_temperatures(mass, scale, every):
    cfg = wca_config(40, 7, (37.0, 29.0), srd=True, seed=2)
    pos, vel = initial_state(cfg, seed=2, layout="rows")
    vel[:, :3] *= np.float32(scale)
    vel[::every, 3] = mass
    with nwgb.System(cfg) as s:
        s.set_array(abi.NW_POSITION, pos)
        s.set_array(abi.NW_VELOCITY, vel)
        got = s.observe()
    nb = cfg.n_beads
    for k, v in (("bead_temperature", vel[:nb]), ("solvent_temperature", vel[nb:])):
        with np.errstate(invalid="ignore"):
            want = obs.temperature(v, cfg.dim)
        if np.isnan(want):
            assert np.isnan(got[k]), k
        else:
            magnitude = obs.temperature(np.abs(v), cfg.dim)  # double sums in another order
            assert got[k] == want or abs(got[k] - want) <= 1e-12 * magnitude, (k, got[k], want)
