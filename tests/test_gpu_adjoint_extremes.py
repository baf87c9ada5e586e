"""Gradients whose terms are infinite or beyond the ordinary range of single
precision: what sums in double precision give."""
import numpy as np
import pytest
import torch

from nwgb.adjoint import Rollout
from nwgb.init import initial_state, wca_config

pytestmark = pytest.mark.gpu

THETA = [1.0, 10.0, 57.0, 0.5]


def _gradients(precision, wp, wv, horizon, L=10):
    cfg = wca_config(40, L, (40.0, 30.0), seed=3)
    pos, vel = initial_state(cfg, seed=3, layout="rows")
    ro = Rollout(cfg, 1, horizon, 2, precision)
    ro.set_state(torch.from_numpy(pos), torch.from_numpy(vel))
    ro.forward(THETA)
    return np.array(ro.backward(wp.cuda(), wv.cuda()))


def _upstream(n, seed=1):
    g = torch.Generator().manual_seed(seed)
    w = [torch.randn(n, 4, generator=g) for _ in range(2)]
    for x in w:
        x[:, 2:] = 0.0
    return w


@pytest.mark.parametrize("value", [float("inf"), -float("inf")])
@pytest.mark.parametrize("bead", [0, 390])
def test_infinite_terms(bead, value):
    """An infinite gradient at the first bead of a worm, which has one bond: the
    terms of k_bend, k_bond and F_act are infinite with a sign, not undefined."""
    wp, wv = _upstream(400)
    wp[bead, 0] = value
    got, want = (_gradients(p, wp, wv, 2) for p in (32, 64))
    assert np.isinf(want[1:]).all()
    assert np.array_equal(got[1:], want[1:])
    assert abs(got[0] - want[0]) <= 1e-5 * abs(want[0]) + 1e-12


@pytest.mark.parametrize("exponent", [85, 104, 110, 116])
@pytest.mark.parametrize("some", [False, True])
def test_large_terms(exponent, some):
    """Scaling the upstream gradients by a power of two, all or some of them,
    scales the terms exactly, so the sums stay the same up to the largest terms
    (46 bits of a sum of 4,000 terms: 1e-9)."""
    wp, wv = _upstream(400)
    f = 2.0 ** exponent
    one = torch.ones(400, 1)
    if some:
        one[::7] = 2.0 ** -40
    base = _gradients(32, wp * one, wv * one, 4)
    got = _gradients(32, wp * one * f, wv * one * f, 4)
    assert np.isfinite(base).all() and np.abs(base).max() > 0
    assert np.abs(got / f - base).max() <= 1e-9 * np.abs(base).max()
