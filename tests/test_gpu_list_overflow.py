"""A three-dimensional bead with more neighbours than its list holds: the
overflow is reported, the update that builds the lists takes all pairs, and
the list keeps the first ones in the order of the scan (cells in z, y, x
order, each cell's beads by index)."""
import numpy as np
import pytest

import nwgb
from nwgb import abi

pytestmark = pytest.mark.gpu

CAP, SKIN = 4, 0.3


def _system():
    n = 8
    c = abi.default_config(abi.NW_MODEL_WCA_WORMS, n ** 3, 1, (10, 10, 10), False)
    c.kT, c.gamma, c.activity, c.dt, c.seed = 0.0, 0.0, 0.0, 0.001, 1
    c.neighbor_capacity, c.neighbor_skin = CAP, SKIN
    rng = np.random.default_rng(2)
    g = np.stack(np.meshgrid(*[np.arange(n)] * 3, indexing="ij"), -1).reshape(-1, 3)
    pos, vel = np.zeros((n ** 3, 4), np.float32), np.zeros((n ** 3, 4), np.float32)
    # 1.05 apart: six neighbours within the cut-off; beads in random order
    pos[:, :3] = 1.2 + 1.05 * rng.permutation(g) + rng.uniform(-0.02, 0.02, (n ** 3, 3))
    pos[:, :3] += np.array([c.origin[a] for a in range(3)])
    pos[:, 3], vel[:, 3] = c.radius, 1.0
    return c, pos, vel


def _pairs(c, r):
    """Every pair's separation (minimum image) and distance, in doubles."""
    box = np.array([c.box[a] for a in range(3)], np.float64)
    d = r[None, :, :].astype(np.float64) - r[:, None, :]
    d -= box * np.rint(d / box)
    return d, np.sqrt((d * d).sum(-1))


def _force(d, q):
    with np.errstate(divide="ignore", invalid="ignore"):
        f = -24.0 * (2.0 * q ** -14 - q ** -8)
    return np.where((q > 0) & (q <= 1.12246205), f, 0.0)[..., None] * d


def _lists(c, r):
    """The first CAP neighbours within the list radius in scan order."""
    rl = 1.12246205 + SKIN
    box, org = (np.array([x[a] for a in range(3)], np.float64) for x in (c.box, c.origin))
    G = np.floor(box / (rl * 1.0001)).astype(int)
    cell = np.floor((r - org) * (G / box)).astype(int) % G
    of = {}
    for i, k in enumerate(map(tuple, cell)):
        of.setdefault(k, []).append(i)
    _, q = _pairs(c, r)
    out, most = [], 0
    for i in range(len(r)):
        found = []
        for z in (-1, 0, 1):
            for y in (-1, 0, 1):
                for x in (-1, 0, 1):
                    k = tuple((cell[i] + (x, y, z)) % G)
                    found += [j for j in of.get(k, []) if j != i and q[i, j] <= rl]
        most = max(most, len(found))
        out.append(found[:CAP])
    assert most > CAP
    return out


def test_overflowing_lists():
    c, pos, vel = _system()
    with nwgb.System(c) as s:
        s.set_array(abi.NW_POSITION, pos)
        s.set_array(abi.NW_VELOCITY, vel)
        s.step(1)
        f1, r1 = s.get_array(abi.NW_FORCE)[:, :3], s.get_array(abi.NW_POSITION)[:, :3]
        assert s.error_word() & abi.NW_EFLAG_NEIGHBOR_OVERFLOW
        s.step(1)
        f2, r2 = s.get_array(abi.NW_FORCE)[:, :3], s.get_array(abi.NW_POSITION)[:, :3]
    # pair forces of up to 10 epsilon and single rounding: 1e-6 relative of each
    # (positions of order 10 to 5e-7, times a stiffness of 300: 2e-4)
    d, q = _pairs(c, r1)
    assert np.abs(f1 - _force(d, q).sum(1)).max() < 1e-3
    d, q = _pairs(c, r2)
    F = _force(d, q)
    want = np.array([F[i, j].sum(0) for i, j in enumerate(_lists(c, r1))])
    assert np.abs(want - F.sum(1)).max() > 1.0  # pairs are missing
    assert np.abs(f2 - want).max() < 1e-3
