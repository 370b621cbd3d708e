"""The step entry's state arrays keep their meaning whatever their layout
(no device needed: the library call is replaced)."""

import numpy as np

import eisenjoch_b200 as E
from eisenjoch_b200 import placer


class _Lib:
    def eplace_stage_step(self, handle, it, *args):
        return 0


def test_step_state_layouts():
    n = 7
    nl = E.Netlist(num_cells=n, net_offsets=np.array([0, 2], np.uint32), pin_cell=np.array([0, 1], np.uint32))
    ctx = placer.PlacementContext.__new__(placer.PlacementContext)
    ctx.netlist, ctx.chip, ctx._lib, ctx.handle = nl, E.Chip(4, 4), _Lib(), None
    f = np.arange(n, dtype=np.float32)
    state = dict(x=f, y=f.astype(np.float64), x_prev=list(f), y_prev=np.arange(2 * n, dtype=np.float32)[::2],
                 gprev_x=np.arange(n + 3, dtype=np.float32), gprev_y=f.reshape(n, 1))
    want = {k: np.array(v, np.float32) for k, v in state.items()}
    z = np.zeros(n, np.float32)
    field = np.zeros((4, 4), np.float32)
    ctx.step(0, z, z, z, z, field, field, state, [0.0, 0.0, 0.1, 0.1])
    for k, v in state.items():
        assert v.dtype == np.float32 and np.array_equal(v, want[k]) and v.shape == want[k].shape, k
    assert state["x"] is not f  # the caller's array is not the one that is updated
