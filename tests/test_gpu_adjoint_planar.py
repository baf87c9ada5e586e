"""Two-dimensional rollouts away from what their two-component kernels assume:
they are computed with all three components then."""
import numpy as np
import pytest
import torch

from nwgb.adjoint import Rollout
from nwgb.init import initial_state, wca_config

pytestmark = pytest.mark.gpu

THETA = [1.0, 10.0, 57.0, 0.5]


def _rollout(cfg, precision, horizon=4):
    pos, vel = initial_state(cfg, seed=3, layout="rows")
    ro = Rollout(cfg, 1, horizon, 3, precision)
    ro.set_state(torch.from_numpy(pos), torch.from_numpy(vel))
    ro.forward(THETA)
    return ro


@pytest.mark.parametrize("precision", [32, 64])
@pytest.mark.parametrize("origin_z", [2.5, -7.25, 0.0])
def test_boxes_without_the_plane(origin_z, precision):
    """A box whose z range does not hold 0 wraps the beads by one box an update."""
    cfg = wca_config(12, 6, (20.0, 16.0), seed=3)
    cfg.origin[2] = origin_z
    z, lo, L = 0.0, cfg.origin[2], cfg.box[2]
    for _ in range(4):
        z += L if z < lo else -L if z > lo + L else 0.0
    assert (z != 0.0) == (origin_z != 0.0)
    got = _rollout(cfg, precision).final_state_f64()[0].cpu().numpy()
    assert np.abs(got[:, 2] - z).max() < 1e-5
    cfg.origin[2] = 0.0
    flat = _rollout(cfg, precision).final_state_f64()[0].cpu().numpy()
    assert np.abs(got[:, :2] - flat[:, :2]).max() < (1e-4 if precision == 32 else 1e-12)


@pytest.mark.parametrize("precision", [32, 64])
@pytest.mark.parametrize("value", [float("nan"), float("inf"), 1e30])
@pytest.mark.parametrize("which", [0, 1])
def test_upstream_gradients_off_the_plane(which, value, precision):
    """Upstream z gradients of a plane's beads reach the parameters times the
    zero z components of the forces: finite ones not at all, others as NaN."""
    cfg = wca_config(12, 6, (20.0, 16.0), seed=3)
    ro = _rollout(cfg, precision)
    g = torch.Generator().manual_seed(2)
    w = [torch.randn(72, 4, generator=g).cuda() for _ in range(2)]
    for x in w:
        x[:, 2:] = 0.0
    base = np.array(ro.backward(*w))
    w[which][31, 2] = value  # inside a worm: bending, bonds and drive
    got = np.array(ro.backward(*w))
    if np.isfinite(value):
        assert np.array_equal(got, base)
    else:
        assert np.isnan(got[1:]).all()
    w[which][31, 2] = 0.0
    assert np.array_equal(np.array(ro.backward(*w)), base)
