"""Order parameters of states with positions that are not numbers: a bead
without a tangent of positive length counts as having none."""
import numpy as np
import pytest

import nwgb
from nwgb import abi
from nwgb.init import initial_state, wca_config

import observables_oracle as obs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("min_image", [False, True])
@pytest.mark.parametrize("axes", [(0,), (1,), (2,), (0, 1), (0, 1, 2)])
def test_beads_at_nan_have_no_tangents(axes, min_image):
    cfg = wca_config(40, 7, (37.0, 29.0), seed=2)
    pos, vel = initial_state(cfg, seed=2, layout="rows")
    for bead in (24, 105, 200):  # inside, at the head of and inside a worm
        pos[bead, list(axes)] = np.nan
    with nwgb.System(cfg) as s:
        s.set_array(abi.NW_POSITION, pos)
        s.set_array(abi.NW_VELOCITY, vel)
        got = s.observe(min_image=min_image)
    with np.errstate(invalid="ignore"):
        t = obs.tangents(pos, 7, [float(cfg.box[0]), float(cfg.box[1]), 0.0] if min_image else None)
    t[np.isnan(t).any(axis=1)] = 0.0
    want = obs.order_parameters(t)
    assert got["n_tangents"] == want["n_tangents"] < 278
    for k in ("s_q3", "s_2d", "polar"):  # float32 tangents on both sides
        assert abs(got[k] - want[k]) < 1e-6, (k, got[k], want[k])
