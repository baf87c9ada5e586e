"""What this engine is measured on: the calls that its users make, over the
sizes and options they run.

A case is one kind of call:
  worms       a simulation loop's call: `steps` updates of a worm system, then
              the frame that the loop reads (2D or 3D, with or without the SRD
              solvent, periodic or as a channel between walls)
  round_trip  a program that owns the state on the host: upload positions and
              velocities, one update, read both back
  dem         the reference's own force model (REF_DEM) with its SRD solvent
  batch       many replicas of uneven size stepped together
  adjoint     a differentiable rollout, forward and backward
  analysis    the analysis of one frame: order parameters, defects, solvent
              temperatures
Initial states are worms laid out without overlaps (turned patches for dilute
planar systems, rows otherwise) with Maxwell-Boltzmann velocities, all drawn
from the seed.  `exact` restates the step, its adjoint and the order
parameters in torch at 64 bits.
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.abspath("nematic-worms_gb300"))

import nwgb  # noqa: E402
from nwgb import abi  # noqa: E402
from nwgb.adjoint import Rollout, rollout  # noqa: E402
from nwgb.batch import Batch  # noqa: E402
from nwgb.init import batch_configs, wca_config  # noqa: E402


def listed():
    return [
        # the small 2D system (400 x 10 beads) in a simulation loop that
        # looks at every hundredth state: launches and their gaps
        dict(name="small_2d_100_updates", kind="worms", dim=2, filaments=400, beads=10, packing=0.314, steps=100),
        # the smallest call: one update of that system by a host program that
        # feeds and reads the state every time
        dict(name="small_2d_round_trip", kind="round_trip", dim=2, filaments=400, beads=10, packing=0.314),
        # an odd-sized 3D system with Langevin noise (the three-component path)
        dict(name="odd_3d", kind="worms", dim=3, filaments=1531, beads=17, packing=0.15, steps=20),
        # passive worms in SRD solvent in a channel (walls in y), odd sizes,
        # every frame read back whole: the smaller solvent runs
        dict(name="channel_srd_frames", kind="worms", dim=2, filaments=1111, beads=9, packing=0.26, steps=10, srd=True,
             walls=True, activity=0.0, frame=True),
        # the headline workload: 400,000 beads and 4,000,000 solvent
        # particles, one SRD period per call
        dict(name="srd_400k", kind="worms", dim=2, filaments=20000, beads=20, packing=0.314159, steps=10, srd=True),
        # the same workload with the bead state owned by the host
        dict(name="srd_400k_round_trip", kind="round_trip", dim=2, filaments=20000, beads=20, packing=0.314159,
             srd=True),
        # the large dense system without solvent
        dict(name="dense_2m", kind="worms", dim=2, filaments=100000, beads=20, packing=0.8, steps=40, activity=1.0),
        # the reference's force model on its feasible stand-in of the headline
        # workload: 400,000 beads on 1024 x 1024 cells, 2.6M solvent particles
        dict(name="dem_srd_400k", kind="dem", filaments=20000, beads=20, grid=1024, steps=5),
        # a parameter sweep: 64 replicas of 50 - 2,000 worms of 5 - 30 beads
        dict(name="batch_64_uneven", kind="batch", replicas=64, worms=2000, beads=30, steps=20),
        # gradients of a loss on the final state: 64 x 4,000 beads, 200 steps
        dict(name="adjoint_64x4k", kind="adjoint", replicas=64, filaments=400, beads=10, packing=0.314, horizon=200,
             segment=20, precision=32),
        # the same at double precision on a small odd system
        dict(name="adjoint_f64_odd", kind="adjoint", replicas=5, filaments=123, beads=11, packing=0.3, horizon=50,
             segment=20, precision=64),
        # the analysis of one frame of the headline workload
        dict(name="analysis_400k", kind="analysis", filaments=20000, beads=20, packing=0.314159, srd=True),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["worms", "worms", "worms", "worms", "round_trip", "dem", "batch", "adjoint", "analysis"])
    L = rng.randint(5, 30)
    if kind == "worms":
        dim = rng.choice([2, 2, 2, 3])
        srd = dim == 2 and rng.random() < 0.5
        nf = max(3, _log(rng, 2000, 400000 if srd else 1500000 if dim == 2 else 200000) // L)
        phi = rng.uniform(0.12, 0.32) if srd else rng.uniform(0.05, 0.2) if dim == 3 else rng.uniform(0.2, 0.75)
        walls = dim == 2 and rng.random() < 0.25
        return dict(kind=kind, dim=dim, filaments=nf, beads=L, packing=phi, steps=10 if srd else rng.randint(1, 40),
                    srd=srd, walls=walls, activity=rng.uniform(0.0, 1.0),
                    frame=bool(srd and nf * L / phi < 400000 and rng.random() < 0.5))
    if kind == "round_trip":
        nf = max(3, _log(rng, 2000, 400000) // L)
        return dict(kind=kind, dim=2, filaments=nf, beads=L, packing=rng.uniform(0.15, 0.32), srd=rng.random() < 0.5)
    if kind == "dem":
        grid = rng.choice([128, 256, 512, 1024])
        return dict(kind=kind, filaments=max(3, int(rng.uniform(0.1, 0.3) * grid * grid / L)), beads=L, grid=grid, steps=5)
    if kind == "batch":
        return dict(kind=kind, replicas=rng.randint(3, 64), worms=_log(rng, 60, 2000), beads=rng.randint(6, 30),
                    steps=rng.randint(2, 20))
    if kind == "adjoint":
        return dict(kind=kind, replicas=rng.randint(1, 32), filaments=_log(rng, 40, 400), beads=rng.randint(3, 20),
                    packing=rng.uniform(0.15, 0.4), horizon=rng.randint(20, 90), segment=rng.randint(8, 20),
                    precision=rng.choice([32, 32, 64]))
    return dict(kind=kind, filaments=max(8, _log(rng, 4000, 400000) // L), beads=L, packing=rng.uniform(0.15, 0.32),
                srd=rng.random() < 0.5)


# ---- configurations and initial states -------------------------------------------


def _config(case, seed):
    kind, nf, L = case["kind"], case.get("filaments", 0), case["beads"]
    if kind == "dem":
        G = case["grid"]
        c = abi.default_config(abi.NW_MODEL_REF_DEM, nf, L, (G, G, 1), True)
        c.bond_r0, c.bend_k, c.activity, c.gamma = 0.8, 10.0, 0.5, 2.0
        c.kT = c.srd_kT = 0.1
    elif case.get("dim", 2) == 3:
        edge = (nf * L * math.pi / 6.0 / case["packing"]) ** (1.0 / 3.0) / 1.12246205
        g = max(int(math.ceil(edge)), int(math.ceil((L * 0.8 + 1.0) / 1.12246205)) + 1)
        c = abi.default_config(abi.NW_MODEL_WCA_WORMS, nf, L, (g, g + 1, g + 2), False)
        c.activity = case.get("activity", 0.5)
    else:
        side = math.sqrt(nf * L * math.pi / 4.0 / case["packing"])
        if kind == "analysis" or case.get("srd"):
            side = float(round(side))
        c = wca_config(nf, L, (side, side), srd=bool(case.get("srd")), activity=case.get("activity", 0.5))
    if case.get("walls"):
        c.boundary[1] = abi.NW_WALL
    c.seed = seed
    return c


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) * 2654435761 % (1 << 62))
    return g


def _rand(g, *shape):
    return torch.rand(*shape, generator=g, device="cuda", dtype=torch.float64)


def _randn(g, *shape):
    return torch.randn(*shape, generator=g, device="cuda", dtype=torch.float64)


def _rows(c, g):
    """Worms along x on a lattice of rows, polarity and a little offset by draw."""
    M, L, dim = c.num_filaments, c.filament_size, c.dim
    box = [c.box[a] for a in range(3)]
    sp = c.bond_r0
    length = (L - 1) * sp
    wall = 1.1 if c.boundary[1] != abi.NW_PERIODIC else 0.0
    per = max(1, int(box[0] // (length + 1.0)))
    lines = -(-M // per)
    nz = max(1, int(box[2] // 1.13)) if dim == 3 else 1
    ny = -(-lines // nz)
    w = torch.randperm(per * ny * nz, generator=g, device="cuda")[:M]
    col, iy, iz = w % per, (w // per) % ny, w // (per * ny)
    sy, sz = (box[1] - wall) / ny, box[2] / nz
    sign = torch.where(_rand(g, M) < 0.5, 1.0, -1.0).double()
    x = (col + 0.5) * (box[0] / per) + (iy % 2) * (0.5 * box[0] / per)
    y = 0.5 * wall + (iy + 0.5) * sy + (_rand(g, M) - 0.5) * min(0.02, 0.2 * sy)
    z = (iz + 0.5) * sz + (_rand(g, M) - 0.5) * min(0.02, 0.2 * sz) if dim == 3 else torch.full_like(y, 0.5 * box[2])
    t = (torch.arange(L, device="cuda") - (L - 1) / 2.0) * sp
    p = torch.stack([x[:, None] + sign[:, None] * t, y[:, None].expand(M, L), z[:, None].expand(M, L)], -1)
    return p.reshape(-1, 3)


def _patches(c, g):
    """Straight worms in parallel patches, each patch turned to an angle by
    draw; None where the box has no room for such patches."""
    M, L = c.num_filaments, c.filament_size
    sp, pitch = c.bond_r0, 1.13
    length = (L - 1) * sp + 1.0
    wall = 1.1 if c.boundary[1] != abi.NW_PERIODIC else 0.0
    for k in range(1, 64):
        rho = math.hypot(length / 2.0, k * pitch / 2.0)
        nx, ny = int(c.box[0] // (2.0 * rho + 0.05)), int((c.box[1] - wall) // (2.0 * rho + 0.05))
        if nx * ny * k >= M:
            break
    else:
        return None
    sites = torch.randperm(nx * ny, generator=g, device="cuda")[: -(-M // k)]
    sx, sy = c.box[0] / nx, (c.box[1] - wall) / ny
    jit = (_rand(g, len(sites), 2) - 0.5) * torch.tensor([sx - 2 * rho, sy - 2 * rho], device="cuda", dtype=torch.float64)
    ang = _rand(g, len(sites)) * (2.0 * math.pi)
    cx = (sites // ny + 0.5) * sx + jit[:, 0]
    cy = 0.5 * wall + (sites % ny + 0.5) * sy + jit[:, 1]
    w = torch.arange(M, device="cuda")
    s, r = w // k, w % k
    d = torch.stack([torch.cos(ang), torch.sin(ang)], -1)[s]
    n = torch.stack([-d[:, 1], d[:, 0]], -1)
    sign = torch.where(_rand(g, M) < 0.5, 1.0, -1.0).double()
    off = (r - (k - 1) / 2.0) * pitch
    t = (torch.arange(L, device="cuda") - (L - 1) / 2.0) * sp
    ctr = torch.stack([cx[s], cy[s]], -1) + off[:, None] * n
    p = ctr[:, None, :] + sign[:, None, None] * t[None, :, None] * d[:, None, :]
    z = torch.full((M, L, 1), 0.5 * c.box[2], device="cuda", dtype=torch.float64)
    return torch.cat([p, z], -1).reshape(-1, 3)


def _state(c, seed):
    """Positions and velocities of a configuration, float4 on the device."""
    g = _gen(seed)
    nb, ns = c.num_filaments * c.filament_size, c.num_solvent if c.srd_enabled else 0
    planar = c.dim == 2 or c.grid[2] == 1
    p = _patches(c, g) if planar else None
    if p is None:
        p = _rows(c, g)
    box = torch.tensor([c.box[a] for a in range(3)], device="cuda", dtype=torch.float64)
    org = torch.tensor([c.origin[a] for a in range(3)], device="cuda", dtype=torch.float64)
    per = torch.tensor([c.boundary[a] == abi.NW_PERIODIC for a in range(3)], device="cuda")
    p = torch.where(per, torch.remainder(p, box), p) + org
    dims = 2 if planar else 3
    pos = torch.zeros(nb + ns, 4, device="cuda")
    vel = torch.zeros(nb + ns, 4, device="cuda")
    pos[:nb, :dims] = p[:, :dims].float()
    pos[:nb, 3], vel[:nb, 3] = c.radius, c.mass
    v = _randn(g, nb, dims) * math.sqrt(c.kT / c.mass)
    vel[:nb, :dims] = (v - v.mean(0)).float()
    if ns:
        pos[nb:, :dims] = (org + _rand(g, ns, 3) * box)[:, :dims].float()
        v = _randn(g, ns, dims) * math.sqrt(c.srd_kT / c.solvent_mass)
        vel[nb:, :dims] = (v - v.mean(0)).float()
        vel[nb:, 3] = c.solvent_mass
    return pos, vel


# ---- the calls ----------------------------------------------------------------------


class _Device:
    """A device array of the engine, as torch takes it; the array lives as
    long as `owner`."""

    def __init__(self, owner, ptr, shape, kind):
        self.owner = owner
        self.__cuda_array_interface__ = dict(shape=shape, typestr=kind, data=(ptr, False), version=3, strides=None)


class _Views:
    """Tensors over the arrays of a system or batch, which stays alive while
    any of them does."""

    def __init__(self, owner):
        self.owner, self.of = owner, {}

    def get(self, ptr, shape, kind="<f4"):
        t = self.of.get(ptr)
        if t is None:
            t = self.of[ptr] = torch.as_tensor(_Device(self.owner, ptr, shape, kind), device="cuda")
            t.owner = self.owner
        return t


def _pinned(n):
    return torch.empty(n, 4, pin_memory=True)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        cfgs = _batch_configs(case, seed)
        b = Batch(cfgs)
        for r, c in enumerate(cfgs):
            pos, vel = _state(c, seed + r)
            b.set_array(r, abi.NW_POSITION, pos.cpu().numpy())
            b.set_array(r, abi.NW_VELOCITY, vel.cpu().numpy())
        return dict(kind=kind, b=b, n=b.total_beads, steps=case["steps"], views=_Views(b))
    c = _config(case, seed)
    if kind == "adjoint":
        R = case["replicas"]
        st = [_state(c, seed * 100 + r) for r in range(R)]
        ro = Rollout(c, R, case["horizon"], case["segment"], case["precision"])
        ro.set_state(torch.cat([s[0] for s in st]), torch.cat([s[1] for s in st]))
        gp, gv = _upstream(case, seed)
        dtype = torch.float64 if case["precision"] == 64 else torch.float32
        return dict(kind=kind, ro=ro, theta=torch.tensor(THETA, dtype=dtype), gp=gp, gv=gv)
    pos, vel = _state(c, seed)
    s = nwgb.System(c)
    s.set_array(abi.NW_POSITION, pos.cpu().numpy())
    s.set_array(abi.NW_VELOCITY, vel.cpu().numpy())
    state = dict(kind=kind, s=s, cfg=c, views=_Views(s), nb=s.n_beads)
    if kind == "analysis":
        rows = s.n_beads // 20 + 64
        state.update(x=np.zeros(rows), y=np.zeros(rows), charge=np.zeros(rows, np.float32), cells=np.zeros(rows, np.int64))
        return state
    n = s.n_beads + (s.n_solvent if case.get("frame") else 0)
    state.update(steps=case.get("steps", 1), frame=bool(case.get("frame")), pos=_pinned(n), vel=_pinned(n))
    state.update(pos_out=state["pos"].numpy(), vel_out=state["vel"].numpy())
    state["force"] = state["views"].get(s.device_ptr(abi.NW_FORCE), (s.n_beads, 4))
    if kind == "round_trip":
        a, b = _pinned(n), _pinned(n)
        a.copy_(pos[:n])
        b.copy_(vel[:n])
        state.update(pos_in=a.numpy(), vel_in=b.numpy(), keep=(a, b))
    elif s.n_solvent:
        state["mean"] = state["views"].get(s.device_ptr(abi.NW_SRD_CELL_MEAN), (s.n_srd_cells, 4))
        state["order"] = state["views"].get(s.device_ptr(abi.NW_SRD_SORTED_INDEX), (s.n_beads + s.n_solvent,), "<i4")
    return state


def run(st):
    kind = st["kind"]
    if kind == "batch":
        b = st["b"]
        b.step(st["steps"])
        out = {}
        for name, which in (("pos", abi.NW_POSITION), ("vel", abi.NW_VELOCITY), ("force", abi.NW_FORCE)):
            p = ctypes.c_void_p()
            abi.check(b.lib.nw_batch_device_array(b.h, which, ctypes.byref(p)))
            out[name] = st["views"].get(p.value, (st["n"], 4))
        return out
    if kind == "adjoint":
        theta = st["theta"].clone().requires_grad_(True)
        pos, vel = rollout(theta, st["ro"])
        torch.autograd.backward((pos, vel), (st["gp"], st["gv"]))
        return dict(pos=pos.detach(), vel=vel.detach(), grad=theta.grad)
    s = st["s"]
    if kind == "analysis":
        out = {"order": s.observe()}
        d = s.find_defects(2.0, max_defects=len(st["x"]))
        for k in ("x", "y", "charge", "cells"):  # the frame's row of a table of frames
            st[k][: len(d)] = d[k]
            st[k][len(d):] = 0
        out["defects"] = {k: st[k] for k in ("x", "y", "charge", "cells")}
        if s.n_solvent:
            out["temperatures"] = s.srd_temperature_histogram(1.0, 64).astype(np.int64)
        return out
    if kind == "round_trip":
        s.set_array_async(abi.NW_POSITION, st["pos_in"])
        s.set_array_async(abi.NW_VELOCITY, st["vel_in"])
        s.step(1)
        s.get_array_async(abi.NW_POSITION, st["pos_out"])
        s.get_array_async(abi.NW_VELOCITY, st["vel_out"])
        return dict(pos=st["pos"], vel=st["vel"], force=st["force"])
    s.step(st["steps"])
    s.get_array_async(abi.NW_POSITION, st["pos_out"])
    out = dict(pos=st["pos"], force=st["force"])
    if st["frame"]:
        s.get_array_async(abi.NW_VELOCITY, st["vel_out"])
        out["vel"] = st["vel"]
    else:
        out["vel"] = st["views"].get(s.device_ptr(abi.NW_VELOCITY), (st["nb"], 4))
    if s.n_solvent:
        out["mean"], out["order"] = st["mean"], st["order"]
    return out


def _batch_configs(case, seed):
    cfgs = batch_configs(case["replicas"], seed=11, worms=(50, case["worms"]), beads=(5, case["beads"]))
    for r, c in enumerate(cfgs):
        c.seed = seed + r
    return cfgs


THETA = [1.1, 8.0, 50.0, 0.8]  # eps, k_bend, k_bond, F_act


def _upstream(case, seed):
    n = case["replicas"] * case["filaments"] * case["beads"]
    g = _gen(seed + 77)
    gp, gv = _randn(g, n, 4).float(), _randn(g, n, 4).float()
    gp[:, 2:], gv[:, 2:] = 0.0, 0.0
    return gp / math.sqrt(n), gv / math.sqrt(n)


def work(case):
    """Per bead and update: position, velocity and force read and written
    (96 bytes) and about 400 operations (bonds, bending, a few pairs, noise);
    per solvent particle and collision: position and velocity read and
    written (64 bytes) and about 60 operations."""
    kind = case["kind"]
    if kind == "batch":  # the mean of the drawn sizes
        n = case["replicas"] * (50 + case["worms"]) / 2 * (5 + case["beads"]) / 2
        return {"bytes": 96.0 * n * case["steps"], "flops": 400.0 * n * case["steps"]}
    n = case["filaments"] * case["beads"]
    if kind == "adjoint":
        n *= case["replicas"] * case["horizon"]
        w = case["precision"] // 32
        return {"bytes": 3.0 * 96.0 * w * n, "flops": 2000.0 * n}
    if kind == "dem":
        ns = 10 * (case["grid"] // 2) ** 2
        return {"bytes": 96.0 * n * case["steps"] + 64.0 * ns, "flops": 600.0 * n * case["steps"] + 60.0 * ns}
    ns = 4 * round(math.sqrt(n * math.pi / 4.0 / case["packing"])) ** 2 if case.get("srd") else 0
    if kind == "analysis":
        return {"bytes": 2 * 16.0 * n + 16.0 * n + 32.0 * ns, "flops": 60.0 * n + 20.0 * ns}
    if kind == "round_trip":
        return {"bytes": 160.0 * n + 6.4 * ns, "flops": 400.0 * n + 6.0 * ns}
    return {"bytes": 96.0 * n * case["steps"] + 64.0 * ns, "flops": 400.0 * n * case["steps"] + 60.0 * ns}


# ---- the same in 64 bits ----------------------------------------------------------------


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        outs = [_exact_worms(c, seed + r, case["steps"]) for r, c in enumerate(_batch_configs(case, seed))]
        return {k: torch.cat([o[k] for o in outs]) for k in ("pos", "vel", "force")}
    c = _config(case, seed)
    if kind == "adjoint":
        return _exact_adjoint(case, c, seed)
    if kind == "analysis":
        out = {"order": _exact_order(c, seed), "defects": dict(x=None, y=None, charge=None, cells=None)}
        if c.srd_enabled:
            out["temperatures"] = None
        return out
    out = _exact_worms(c, seed, case.get("steps", 1), dem=kind == "dem", frame=bool(case.get("frame")))
    if kind == "round_trip":
        return {k: out[k] for k in ("pos", "vel", "force")}
    return out


def _philox(i, step, stream, k0, k1):
    """Philox4x32-10 (Salmon et al., SC'11) on int64 tensors of 32-bit words."""
    m = 0xFFFFFFFF
    x = [i & m, torch.full_like(i, step & m), torch.full_like(i, (step >> 32) & m), torch.full_like(i, stream)]
    for r in range(10):
        if r:
            k0, k1 = (k0 + 0x9E3779B9) & m, (k1 + 0xBB67AE85) & m
        a, b = x[0] * 0xD2511F53, x[2] * 0xCD9E8D57
        x = [((b >> 32) & m) ^ x[1] ^ k0, b & m, ((a >> 32) & m) ^ x[3] ^ k1, a & m]
    return x


def _u01(x):
    return ((x >> 9).double() + 0.5) / 8388608.0


def _normals(x, dim):
    out = []
    for a, b in ((x[0], x[1]), (x[2], x[3])):
        r, t = torch.sqrt(-2.0 * torch.log(_u01(a))), 2.0 * math.pi * _u01(b)
        out += [r * torch.cos(t), r * torch.sin(t)]
    if dim < 3:
        out[2] = torch.zeros_like(out[2])
    return torch.stack(out[:3], -1)


class _Sys:
    """The worm step in 64 bits on (n, 3) tensors."""

    def __init__(self, c, theta=None):
        d = dict(device="cuda", dtype=torch.float64)
        self.c, self.L, self.dt = c, c.filament_size, float(c.dt)
        self.n = c.num_filaments * c.filament_size
        self.box = torch.tensor([c.box[a] for a in range(3)], **d)
        self.org = torch.tensor([c.origin[a] for a in range(3)], **d)
        self.per = torch.tensor([c.boundary[a] == abi.NW_PERIODIC for a in range(3)], device="cuda")
        self.span = torch.where(self.per, self.box, torch.full_like(self.box, 1e30))
        s2 = 2.0 * c.gamma * c.kT / (self.dt if c.noise_dt_scaling else 1.0)
        self.sigma = math.sqrt(s2)
        self.theta = theta if theta is not None else [float(c.lj_epsilon), float(c.bend_k), float(c.bond_k), float(c.activity)]

    def near(self, d):
        return d - self.span * torch.round(d / self.span)

    def bounds(self, p, v, rad):
        for a in range(3):
            lo, hi = float(self.c.origin[a]), float(self.c.origin[a]) + float(self.c.box[a])
            q = p[:, a]
            if self.c.boundary[a] == abi.NW_PERIODIC:
                q = q + (q < lo) * self.box[a] - (q > hi) * self.box[a]
            else:
                out = (q < lo + rad) | (q > hi - rad)
                v = v.clone()
                v[:, a] = torch.where(out, v[:, a] * float(self.c.boundary_damping), v[:, a])
                q = q.clamp(lo + rad, hi - rad)
            p = torch.cat([p[:, :a], q[:, None], p[:, a + 1:]], 1)
        return p, v

    def chain(self, r, bonds=True):
        """Bending, and with `bonds` the harmonic bonds and the drive."""
        eps, kb, k, fa = self.theta
        x = r.reshape(-1, self.L, 3)
        f = torch.zeros_like(x)
        if self.L < 2:
            return f.reshape(-1, 3)
        b = self.near((x[:, 1:] - x[:, :-1]).reshape(-1, 3)).reshape(-1, self.L - 1, 3)
        d = b.norm(dim=-1, keepdim=True)
        pad = lambda t, lo, hi: torch.nn.functional.pad(t, (0, 0, lo, hi))  # noqa: E731
        if self.L >= 3:
            a, e = b[:, :-1], b[:, 1:]
            da, de = d[:, :-1], d[:, 1:]
            dot = (a * e).sum(-1, keepdim=True)
            A = 1.0 / (da * de)
            fi = -A * (e - a * dot / da ** 2)
            fk = -A * (e * dot / de ** 2 - a)
            f = f + kb * (pad(fi, 0, 2) + pad(-fi - fk, 1, 1) + pad(fk, 2, 0))
        if bonds:
            t = k * (d - float(self.c.bond_r0)) * b / d
            f = f + pad(t, 0, 1) - pad(t, 1, 0) + fa * pad(b / d, 0, 1)
        return f.reshape(-1, 3)

    def cells(self, r, rc):
        dims = [max(1, int(float(self.box[a]) // (rc * 1.0001))) if self.c.grid[a] > 1 else 1 for a in range(3)]
        G = torch.tensor(dims, device="cuda")
        g = torch.floor((r - self.org) / self.box * G).long()
        return torch.where(self.per, g % G, torch.minimum(g.clamp(min=0), G - 1)), dims

    def pairs(self, r, rc):
        """(i, j): every bead j within rc of bead i that takes part in the
        pair force (both directions)."""
        g, G = self.cells(r.detach(), rc)
        return self.from_cells(g, G, lambda i, j: self.close(r, i, j, rc))

    def close(self, r, i, j, rc):
        d = self.near(r[j] - r[i])
        far = (j - i).abs() > self.c.lj_exclude
        return ((d * d).sum(-1) <= rc * rc) & (far | (torch.div(i, self.L, rounding_mode="floor") != torch.div(j, self.L, rounding_mode="floor")))

    def from_cells(self, g, G, keep):
        n = g.shape[0]
        h = (g[:, 2] * G[1] + g[:, 1]) * G[0] + g[:, 0]
        order = torch.argsort(h, stable=True)
        ncell = G[0] * G[1] * G[2]
        cnt = torch.bincount(h, minlength=ncell)
        start = torch.cumsum(cnt, 0) - cnt
        cap = int(cnt.max())
        me = torch.arange(n, device="cuda")
        I, J = [], []
        offs = [sorted({o % Ga if per else o for o in ((-1, 0, 1) if Ga > 1 else (0,))}) for Ga, per in zip(G, self.per.tolist())]
        for oz in offs[2]:
            for oy in offs[1]:
                for ox in offs[0]:
                    q = g + torch.tensor([ox, oy, oz], device="cuda")
                    Gt = torch.tensor(G, device="cuda")
                    q = torch.where(self.per, q % Gt, q)
                    ok = ((q >= 0) & (q < Gt)).all(-1)
                    hq = torch.where(ok, (q[:, 2] * G[1] + q[:, 1]) * G[0] + q[:, 0], 0)
                    for k in range(cap):
                        i = me[ok & (cnt[hq] > k)]
                        j = order[start[hq[i]] + k]
                        m = (i != j) & keep(i, j)
                        I.append(i[m])
                        J.append(j[m])
        return torch.cat(I), torch.cat(J)

    def lj(self, r, ij, rc):
        i, j = ij
        d = self.near(r[j] - r[i])
        q = (d * d).sum(-1, keepdim=True)
        s6 = float(self.c.lj_sigma) ** 6
        iq = 1.0 / q
        w = 24.0 * s6 * (2.0 * s6 * iq ** 7 - iq ** 4) * (q <= rc * rc)
        return torch.zeros_like(r).index_add(0, i, -self.theta[0] * w * d)

    def noise(self, step, seed, first=0, n=None):
        i = torch.arange(n or self.n, device="cuda")
        return self.sigma * _normals(_philox(i, step, 1, seed & 0xFFFFFFFF, (seed >> 32) & 0xFFFFFFFF), self.c.dim)

    def move(self, r, v, F, Fo):
        v = v + 0.5 * self.dt * (F + Fo)
        return (*self.bounds(r + self.dt * v + 0.5 * self.dt ** 2 * F, v, float(self.c.radius)),)


def _axis32(x, origin, cell, box, G, wall, wrap, shift=0.0):
    """Cell index of float32 coordinates, in float32 as a simulation takes it."""
    f = np.float32
    rel = (x + f(shift)) - f(origin)
    if wrap and not wall:
        rel = torch.where(rel >= f(box), rel - f(box), torch.where(rel < 0, rel + f(box), rel))
    g = torch.floor(rel / torch.full_like(rel, float(f(cell)))).long()  # a tensor: torch multiplies by 1 / a scalar
    return g.clamp(0, G - 1) if wall else g % G


def _collide(S, c, step, bpos32, spos32, bv, sv, spos):
    """One SRD collision and the solvent's streaming."""
    nb, ns = bv.shape[0], sv.shape[0]
    G = [int(c.srd_grid[a]) for a in range(3)]
    k0, k1 = int(c.seed) & 0xFFFFFFFF, int(c.seed) >> 32
    x = _philox(torch.zeros(1, dtype=torch.int64, device="cuda"), step, 3, k0, k1)
    h = torch.zeros(nb + ns, dtype=torch.int64, device="cuda")
    for a in (2, 1, 0):
        if G[a] == 1:
            continue
        u = np.float32(float(_u01(x[a])))
        shift = (np.float32(c.srd_shift_lo) + u) * np.float32(c.srd_cell_size[a])
        q = torch.cat([bpos32[:, a], spos32[:, a]])
        g = _axis32(q, c.origin[a], c.srd_cell_size[a], c.box[a], G[a], c.boundary[a] != abi.NW_PERIODIC, True, shift)
        h = h * G[a] + g
    nc = G[0] * G[1] * G[2]
    v = torch.cat([bv, sv])
    m = torch.cat([torch.full((nb, 1), float(c.mass)), torch.full((ns, 1), float(c.solvent_mass))]).cuda().double()
    tot = lambda t: torch.zeros(nc, t.shape[1], device="cuda", dtype=torch.float64).index_add(0, h, t)  # noqa: E731
    if c.srd_thermostat == abi.NW_SRD_THERMO_REF_LAB:
        E = tot(0.5 * m * (v * v).sum(-1, keepdim=True))
        v = v * torch.sqrt(float(c.srd_kT) / E)[h]
    M = tot(m)
    u = tot(m * v) / torch.where(M > 0, M, torch.ones_like(M))
    x = _philox(torch.arange(nc, device="cuda"), step, 4, k0, k1)
    sgn = torch.where(_u01(x[0]) > 0.5, 1.0, -1.0)[h]
    ca, sa = math.cos(float(c.srd_alpha)), math.sin(float(c.srd_alpha)) * sgn
    d = v - u[h]
    rot = torch.stack([d[:, 0] * ca - d[:, 1] * sa, d[:, 0] * sa + d[:, 1] * ca, d[:, 2]], -1)
    turned = torch.arange(nb + ns, device="cuda") >= (0 if c.srd_rotate_beads else nb)
    if c.srd_thermostat == abi.NW_SRD_THERMO_CELL_REL:
        w = turned[:, None].double()
        ke = tot(w * 0.5 * m * (rot[:, :2] ** 2).sum(-1, keepdim=True))
        n = tot(w)
        lam = torch.where((n >= 2) & (ke > 0), torch.sqrt((n - 1) * float(c.srd_kT) / ke), torch.ones_like(ke))[h]
        rot = torch.cat([rot[:, :2] * lam, rot[:, 2:]], -1)
    v = torch.where(turned[:, None], u[h] + rot, v)
    order = torch.argsort(h, stable=True)
    so = order[order >= nb] - nb
    sv, sp = v[nb:][so], spos[so]
    sp, sv = S.bounds(sp + float(c.dt) * c.srd_gap * sv, sv, 0.0)
    return v[:nb], sv, sp, u


def _exact_worms(c, seed, steps, dem=False, frame=False):
    pos, vel = _state(c, seed)
    S = _Sys(c)
    nb = S.n
    r, v = pos[:nb, :3].double(), vel[:nb, :3].double()
    sp, sv = pos[nb:, :3].double(), vel[nb:, :3].double()
    F, Fo = torch.zeros_like(r), torch.zeros_like(r)
    rc, mean = float(c.lj_rcut), None
    # the first update starts from zero forces, so its float32 positions, and
    # with them the cells, are known to the bit
    p32 = pos[:nb, :3] + vel[:nb, :3] * np.float32(c.dt)
    p32, _ = S.bounds(p32.double(), vel[:nb, :3].double(), float(c.radius))
    for n in range(steps):
        r, v = S.move(r, v, F, Fo)
        Fo, F = F, S.chain(r, bonds=not dem)
        cur32 = p32.float() if n == 0 else r.float()
        if not c.srd_enabled:
            F = F + S.noise(n, int(c.seed)) - float(c.gamma) * v
        hit = bool(c.srd_enabled) and n % c.srd_gap == 0
        if hit and n > 0:
            return None  # the solvent's order after a second collision hangs on float32 cell edges
        if dem:
            F = F + _dem_pairs(S, c, r, v, cur32)
        if hit:
            v, sv, sp, mean = _collide(S, c, n, cur32, pos[nb:, :3], v, sv, sp)
        if not dem:
            F = F + S.lj(r, S.pairs(r, rc), rc)

    def f4(x, w):
        return torch.cat([x, torch.full((x.shape[0], 1), float(w), device="cuda", dtype=torch.float64)], 1)

    if frame:
        P = torch.cat([f4(r, c.radius), f4(sp, 0.0)])
        V = torch.cat([f4(v, c.mass), f4(sv, c.solvent_mass)])
    else:
        P, V = f4(r, c.radius), f4(v, c.mass)
    out = dict(pos=P, vel=V, force=f4(F, 0.0))
    if mean is not None:
        out.update(mean=f4(mean, 0.0), order=None)
    return out


def _dem_pairs(S, c, r, v, r32):
    """REF_DEM pair forces: every bead of the 3 x 3 cells around, three times
    (the reference's z offsets on one layer)."""
    G = [int(c.grid[a]) for a in range(3)]
    g = torch.zeros(S.n, 3, dtype=torch.int64, device="cuda")
    for a in range(2):
        g[:, a] = _axis32(r32[:, a], c.origin[a], c.cell_size[a], c.box[a], G[a], False, False)
    i, j = S.from_cells(g, G, lambda i, j: torch.ones_like(i, dtype=torch.bool))
    x = r.reshape(-1, S.L, 3)
    t = torch.zeros_like(x)
    t[:, 1:-1] = S.near((x[:, 2:] - x[:, :-2]).reshape(-1, 3)).reshape(-1, S.L - 2, 3)
    t[:, 0] = S.near(x[:, 1] - x[:, 0])
    t[:, -1] = S.near(x[:, -1] - x[:, -2])
    t = (t / t.norm(dim=-1, keepdim=True)).reshape(-1, 3)
    rel = S.near(r[j] - r[i])
    d = rel.norm(dim=-1, keepdim=True)
    n = rel / d
    same = (i // S.L == j // S.L)[:, None]
    bonded = same & ((i - j).abs() == 1)[:, None]
    rv = v[j] - v[i]
    tv = rv - (rv * n).sum(-1, keepdim=True) * n
    cd = 2.0 * float(c.radius)
    hit = -float(c.spring) * (cd - d) * n + float(c.damping) * rv + float(c.shear) * tv
    f = torch.where(bonded, -float(c.bond_k) * (float(c.bond_r0) - d) * n, torch.where(d < cd, hit, torch.zeros_like(hit)))
    anti = ~same & ((t[i] * t[j]).sum(-1, keepdim=True) < -0.5)
    f = f + torch.where(anti, -float(c.activity) * (t[i] - t[j]) / (2.0 * d), torch.zeros_like(f))
    return 3.0 * torch.zeros_like(r).index_add(0, i, f)


def _exact_adjoint(case, c, seed):
    R, nb = case["replicas"], c.num_filaments * c.filament_size
    st = [_state(c, seed * 100 + r) for r in range(R)]
    theta = torch.tensor(THETA, dtype=torch.float32 if case["precision"] == 32 else torch.float64).double().cuda().requires_grad_(True)
    gp, gv = _upstream(case, seed)
    P, V = [], []
    loss = 0.0
    S = _Sys(c, theta)
    rc = float(c.lj_rcut)
    skin = float(c.neighbor_skin) if c.neighbor_skin > 0 else 0.3 * float(c.lj_sigma)
    r = torch.cat([s[0] for s in st])[:, :3].double()
    v = torch.cat([s[1] for s in st])[:, :3].double()
    F, Fo = torch.zeros_like(r), torch.zeros_like(r)
    for m in range(case["horizon"]):
        if m % case["segment"] == 0:
            with torch.no_grad():
                ij = [S.pairs(r[k * nb:(k + 1) * nb], rc + skin) for k in range(R)]
                ij = (torch.cat([a + k * nb for k, (a, b) in enumerate(ij)]), torch.cat([b + k * nb for k, (a, b) in enumerate(ij)]))
        r, v = S.move(r, v, F, Fo)
        xi = torch.cat([S.noise(m, int(c.seed) + k) for k in range(R)])
        Fo, F = F, S.chain(r) + S.lj(r, ij, rc) + xi - float(c.gamma) * v
    loss = (r * gp[:, :3].double()).sum() + (v * gv[:, :3].double()).sum()
    grad = torch.autograd.grad(loss, theta)[0]
    w = lambda x, k: torch.cat([x.detach(), torch.cat([s[k] for s in st])[:, 3:].double()], 1)  # noqa: E731
    return dict(pos=w(r, 0), vel=w(v, 1), grad=grad.cpu())


def _exact_order(c, seed):
    pos, vel = _state(c, seed)
    nb, L = c.num_filaments * c.filament_size, c.filament_size
    r = pos[:nb, :3].double()
    i = torch.arange(nb, device="cuda")
    a, b = torch.where(i % L == 0, i, i - 1), torch.where(i % L == L - 1, i, (i + 1).clamp(max=nb - 1))
    d = (r[b] - r[a])[1:-1]
    t = d / d.norm(dim=-1, keepdim=True)
    Q = 1.5 * (t.T @ t) / nb - 0.5 * torch.eye(3, device="cuda", dtype=torch.float64)
    q = t[:, 0] ** 2 + t[:, 1] ** 2
    c2, s2 = ((t[:, 0] ** 2 - t[:, 1] ** 2) / q).mean(), (2 * t[:, 0] * t[:, 1] / q).mean()
    T = lambda v: float((v[:, 3].double() * (v[:, :c.dim].double() ** 2).sum(-1)).mean() / c.dim) if len(v) else 0.0  # noqa: E731
    return dict(s_q3=float(torch.linalg.eigvalsh(Q)[-1]), s_2d=float(torch.hypot(c2, s2)),
                polar=float((t.sum(0) / nb).norm()), bead_temperature=T(vel[:nb]), solvent_temperature=T(vel[nb:]),
                msd=None, n_beads=None, n_tangents=None, n_solvent=None)
