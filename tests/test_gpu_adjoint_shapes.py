"""The adjoint's update kernels at the filament lengths and sizes where their
blocks change: whole filaments of 1 to 300 beads per block, partly filled and
single blocks, segments of one update, against the FP64 torch rollout."""
import numpy as np
import pytest
import torch

import torch_rollout
from nwgb.adjoint import Rollout, rollout
from nwgb.init import initial_state, wca_config

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nf,L,R,H,seg,box", [
    (5, 1, 2, 4, 4, (12.0, 12.0)), (7, 2, 1, 5, 1, (12.0, 14.0)), (9, 3, 2, 6, 5, (14.0, 13.0)),
    (3, 63, 1, 5, 2, (60.0, 9.0)), (10, 64, 2, 3, 3, (70.0, 20.0)), (33, 13, 3, 7, 3, (40.0, 30.0)),
    (2, 257, 1, 4, 3, (215.0, 8.0)),
])
def test_update_blocks_match_the_torch_rollout(nf, L, R, H, seg, box):
    cfg = wca_config(nf, L, box, seed=3)
    st = [initial_state(cfg, seed=20 + r, layout="rows") for r in range(R)]
    pos, vel = (np.concatenate([s[k] for s in st]) for k in (0, 1))
    ro = Rollout(cfg, R, H, seg, 64)
    ro.set_state(torch.from_numpy(pos), torch.from_numpy(vel))
    g = torch.Generator().manual_seed(1)
    wp, wv = (torch.randn(R * nf * L, 4, generator=g, dtype=torch.float64) for _ in range(2))
    wp[:, 2:] = wv[:, 2:] = 0.0
    th = torch.tensor([1.0, 10.0, 57.0, 0.5], dtype=torch.float64, requires_grad=True)
    p, v = rollout(th, ro)
    torch.autograd.backward((p, v), (wp.float().cuda(), wv.float().cuda()))
    p64, v64 = (x.cpu() for x in ro.final_state_f64())
    ref_th = torch.tensor([1.0, 10.0, 57.0, 0.5], dtype=torch.float64, requires_grad=True)
    rp, rv = torch_rollout.rollout(cfg, ref_th, pos, vel, R, H, seg, torch_rollout.noise_table(cfg, R, H))
    (gr,) = torch.autograd.grad((rp[:, :3] * wp.float().double()[:, :3]).sum() + (rv[:, :3] * wv.float().double()[:, :3]).sum(),
                                ref_th, allow_unused=True)
    # double precision on both sides, a handful of updates: rounding only
    assert float((p64[:, :3] - rp.detach()[:, :3]).abs().max()) < 1e-9
    assert float((v64[:, :3] - rv.detach()[:, :3]).abs().max()) < 1e-9
    scale = float(gr.abs().max())
    assert float((th.grad - gr).abs().max()) < 1e-8 * scale + 1e-12


@pytest.mark.parametrize("precision", [32, 64])
def test_replicas_do_not_depend_on_the_block_size(precision):
    """Enough replicas for blocks of 256 threads against two of them alone, in
    blocks of 64: the same states to the bit."""
    cfg = wca_config(300, 20, (180.0, 60.0), seed=4)
    out = []
    for R in (26, 2):
        st = [initial_state(cfg, seed=r, layout="rows") for r in range(R)]
        ro = Rollout(cfg, R, 5, 3, precision)
        ro.set_state(torch.from_numpy(np.concatenate([s[0] for s in st])),
                     torch.from_numpy(np.concatenate([s[1] for s in st])))
        ro.forward([1.0, 10.0, 57.0, 0.5])
        out.append([x[:2 * cfg.n_beads].cpu() for x in ro.final_state_f64()])
    for a, b in zip(*out):
        assert torch.equal(a, b)
