"""Cell lists of a batch's replicas from a few beads to several blocks' share
of them: the same state whatever the number of blocks and threads that build
them, and that of the replica run as a system of its own."""
import numpy as np
import pytest

import nwgb
from nwgb import abi
from nwgb.batch import Batch
from nwgb.init import initial_state, wca_config

pytestmark = pytest.mark.gpu

# beads at which a thread takes more than one: 8 x and 32 x 128, 256 and 512
WORMS = (1, 63, 127, 129, 255, 257, 511, 513, 1023, 1025, 2100, 4200)


def _configs():
    out = []
    for k, nf in enumerate(WORMS):
        side = float(np.sqrt(nf * 8 / 0.35)) + 12.0
        c = wca_config(nf, 8, (side, side), seed=20 + k)
        c.neighbor_skin = 0.05  # several builds in a call
        out.append(c)
    return out


def test_lists_of_replicas_of_many_sizes():
    cfgs = _configs()
    states = [initial_state(c, seed=k, layout="rows") for k, c in enumerate(cfgs)]
    first = None
    for threads in (128, 256, 512):
        with Batch(cfgs) as b:
            b.set_tuning(threads, abi.NW_STRATEGY_VERLET, 0.05)
            for r, (pos, vel) in enumerate(states):
                b.set_array(r, abi.NW_POSITION, pos)
                b.set_array(r, abi.NW_VELOCITY, vel)
            b.step(7)
            b.step(1)
            b.step(5)
            b.sync()
            got = [b.get_array(r, abi.NW_POSITION) for r in range(len(cfgs))]
        first = first or got
        for r, (x, y) in enumerate(zip(first, got)):
            assert np.array_equal(x.view(np.uint32), y.view(np.uint32)), (threads, r)
    for c, (pos, vel), got in zip(cfgs, states, first):
        c.strategy = abi.NW_STRATEGY_VERLET
        with nwgb.System(c) as s:
            s.set_array(abi.NW_POSITION, pos)
            s.set_array(abi.NW_VELOCITY, vel)
            s.step(13)
            want = s.get_array(abi.NW_POSITION)
        # the same pairs in the same order; 13 updates of single rounding
        assert np.abs(got[:, :3] - want[:, :3]).max() < 1e-3
