"""The mixed-precision transform's operand ring: products of fewer K steps than
the ring has stages (the whole sum's loads of the fixed operand are issued
before the kernel before has ended), of as many, and of more, on grids of each
tile shape, against the FP64 oracle.

Tolerance: 1e-4 normwise, the parity tests' bound for this transform.
"""
import numpy as np
import pytest

import eisenjoch_b200 as E
from oracle.oracle import Oracle
from tests.conftest import rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("field_mode", [0, 1])
@pytest.mark.parametrize("bx,by", [(64, 128), (128, 128), (192, 256), (256, 384), (320, 128), (576, 256)])
def test_ring_lengths(bx, by, field_mode):
    n = 4000
    nl, chip = E.synth_netlist(E.SynthSpec(seed=bx + by, num_cells=n, num_nets=n, num_pads=40, width=bx, height=by,
                                           bins_x=bx, bins_y=by, cluster_size=32))
    rng = np.random.default_rng(bx * by)
    x = rng.uniform(0, bx - 1, n).astype(np.float32)
    y = rng.uniform(0, by - 1, n).astype(np.float32)
    orc = Oracle(nl, chip)
    d = orc.density(x, y)
    with E.PlacementContext(nl, chip) as ctx:
        got = [ctx.field(d, dct_mode=E._abi.EPLACE_DCT_BF16X3_TC, want_phi=True, field_mode=field_mode)
               for _ in range(2)]
    want = orc.field(d, 1.0, want_phi=True, field_mode=field_mode)
    for g, again, w in zip(got[0], got[1], want):
        assert rel_err(g, w) <= 1e-4
        assert np.array_equal(g, again)
