"""The single-precision routes of the analysis kernels where they hand over to
double precision: speeds, masses and temperatures at the edges of their
ranges, and beads on grid-cell edges."""
import numpy as np
import pytest

import observables_oracle as obs
import nwgb
from nwgb import abi
from nwgb.init import initial_state, wca_config

pytestmark = pytest.mark.gpu


def _system(nf=40, L=7, box=(37.0, 29.0), seed=2):
    cfg = wca_config(nf, L, box, srd=True, seed=seed)
    pos, vel = initial_state(cfg, seed=seed, layout="rows")
    return cfg, pos, vel


@pytest.mark.parametrize("scale", [0.0, 1e-30, 1e-18, 1e-13, 1e-6, 1.0, 30.0, 1e6, 1e15])
@pytest.mark.parametrize("mass", [1.0, 0.7])
def test_temperatures_at_any_speed(scale, mass):
    cfg, pos, vel = _system()
    vel[:, :3] *= np.float32(scale)
    vel[::3, 3] = mass
    with nwgb.System(cfg) as s:
        s.set_array(abi.NW_POSITION, pos)
        s.set_array(abi.NW_VELOCITY, vel)
        got = s.observe()
    nb = cfg.n_beads
    for k, v in (("bead_temperature", vel[:nb]), ("solvent_temperature", vel[nb:])):
        want = obs.temperature(v, cfg.dim)
        assert abs(got[k] - want) <= 1e-12 * want, (k, got[k], want)


@pytest.mark.parametrize("kT", [1e-4, 0.1, 1.5, 40.0])
@pytest.mark.parametrize("mass", [1.0, 2.5])
def test_histogram_equals_the_fixed_point_sums(kT, mass):
    """Cells of hot, cold and unequal particles, and bins fine enough that many
    temperatures lie next to an edge."""
    cfg, pos, vel = _system(seed=5)
    nb = cfg.n_beads
    vel[:, :2] *= np.float32(np.sqrt(kT / 0.1))
    vel[nb::2, 3] = mass
    with nwgb.System(cfg) as s:
        s.set_array(abi.NW_POSITION, pos)
        s.set_array(abi.NW_VELOCITY, vel)
        for bins, t_max in ((64, 4.0 * kT), (4096, 0.5 * kT), (1, kT)):
            got = s.srd_temperature_histogram(t_max, bins)
            assert np.array_equal(got, _histogram(pos, vel, cfg, t_max, bins)), (bins, t_max)


def _histogram(pos, vel, cfg, t_max, bins):
    """The same integers in numpy: 2^32 fixed point, separately rounded doubles."""
    f = np.float32
    c = np.zeros(len(pos), np.int64)
    for a in (1, 0):
        p = (pos[:, a] + f(0)) - f(cfg.origin[a])
        p = np.where(p >= f(cfg.box[a]), p - f(cfg.box[a]), np.where(p < 0, p + f(cfg.box[a]), p))
        c = c * int(cfg.srd_grid[a]) + np.floor(p / f(cfg.srd_cell_size[a])).astype(np.int64) % int(cfg.srd_grid[a])
    n = int(cfg.srd_grid[0]) * int(cfg.srd_grid[1])
    v = vel.astype(np.float64)
    m = v[:, 3]
    fix = lambda x: np.rint(x * 4294967296.0).astype(np.int64)  # noqa: E731
    M, px, py, ke = (_sum(c, fix(x), n) / 4294967296.0 for x in (m, m * v[:, 0], m * v[:, 1], m * (v[:, 0] ** 2 + v[:, 1] ** 2)))
    cnt = np.bincount(c, minlength=n)
    ok = cnt >= 2
    T = (ke[ok] - (px[ok] ** 2 + py[ok] ** 2) / M[ok]) / (2.0 * (cnt[ok] - 1))
    b = np.floor(T / float(f(t_max)) * bins)
    k = np.where(b < 0, 0, np.minimum(b, bins)).astype(np.int64)
    out = np.zeros(bins + 2, np.uint32)
    np.add.at(out, k, 1)
    out[bins + 1] = ok.sum()
    return out


def _sum(c, x, n):
    s = np.zeros(n, np.int64)
    np.add.at(s, c, x)
    return s


@pytest.mark.parametrize("cs", [2.0, 1.5, 0.7])
def test_defect_grid_with_beads_on_cell_edges(cs):
    """Beads at multiples of the cell edge from the lowest bead, rounded to
    float32 to either side of it, fall into the cells that float64 gives."""
    import defects_oracle as orc

    cs = float(np.float32(cs))  # the device takes the edge as a float
    rng = np.random.default_rng(4)
    n, L = 3000, 6
    cfg = wca_config(n, L, (260.0, 250.0), seed=1)
    c, a = rng.uniform(-110, 110, (n, 1, 2)), rng.uniform(0, 2 * np.pi, (n, 1))
    k = 0.8 * (np.arange(L) - 2.5)
    xy = (c + np.stack([k * np.cos(a), k * np.sin(a)], -1)).reshape(-1, 2).astype(np.float32)
    low = xy.min(axis=0).astype(np.float64)
    for axis in (0, 1):
        edge = low[axis] + np.rint((xy[axis::3, axis] - low[axis]) / cs) * cs
        xy[axis::3, axis] = np.maximum(edge, low[axis])
    pos = np.zeros((n * L, 4), np.float32)
    pos[:, :2] = xy
    with nwgb.System(cfg) as s:
        s.set_array(abi.NW_POSITION, pos)
        got = s.find_defects(cs)
    want = orc.find_defects(pos[:, :3], L, cs)
    assert np.array_equal(got["charge"], want["charge"]) and np.array_equal(got["cells"], want["cells"])
    for f in ("x", "y"):  # mean cell index * edge + origin in doubles: a few ulp of 256
        assert np.abs(got[f] - want[f]).max() < 4 * np.spacing(256.0), f
