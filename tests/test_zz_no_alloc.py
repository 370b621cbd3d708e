"""The allocation-free density entry point (eplace_density_noalloc).

It serves callers that cannot call cudaMalloc: a real-time loop that must
not allocate or wait on the allocator, an application whose device memory is
owned and handed out by another component, code under a fixed device-memory
budget.  They pass device buffers they already own (here the test allocates
them with torch, standing in for such an owner) and the library uses a fixed
array of its own as working memory.

Checked through the C ABI, on two calls in a row each (the second proves the
shared working array is clean between calls):
  * against the regular density entry point: the same map bit for bit (both
    run the same fixed-point scatter), the overlap to 1e-12 relative (its
    FP64 sum may be split over a different number of blocks);
  * against the FP64 oracle: the parity tolerances of the density stage
    (normwise 1e-5, overlap 1e-6 absolute);
  * the 1x1-cell path (half_wh = NULL), an empty design, and the host-side
    rejection of oversized grids and misaligned pointers.
The file is named so that pytest collects it last.
"""

import ctypes

import numpy as np
import pytest

import eisenjoch_b200 as E
from eisenjoch_b200 import _abi
from oracle.oracle import Oracle
from tests.conftest import rel_err

pytestmark = pytest.mark.gpu


def _positions(nl, chip, seed):
    rng = np.random.default_rng(seed)
    n = nl.num_cells
    cx = rng.uniform(0.3, 0.7, 6) * (chip.width - 1)
    cy = rng.uniform(0.3, 0.7, 6) * (chip.height - 1)
    k = rng.integers(0, 6, n)
    x = np.clip(cx[k] + rng.normal(0, chip.width * 0.05, n), 0, chip.width - 1).astype(np.float32)
    y = np.clip(cy[k] + rng.normal(0, chip.height * 0.05, n), 0, chip.height - 1).astype(np.float32)
    return x, y


def _noalloc(torch, nl, chip, x, y, half_d, dens_d, ov_d):
    L = _abi.lib()
    dev = dens_d.device
    pos_d = torch.from_numpy(np.ascontiguousarray(np.stack([x, y], axis=1))).to(dev)
    stream = torch.cuda.current_stream(dev)
    bx, by = chip.bins_x or chip.width, chip.bins_y or chip.height  # 0: one bin per site
    st = L.eplace_density_noalloc(
        ctypes.c_void_p(pos_d.data_ptr() if nl.num_cells else 0),
        ctypes.c_void_p(half_d.data_ptr() if half_d is not None else 0), nl.num_cells, chip.width, chip.height,
        bx, by, ctypes.c_void_p(dens_d.data_ptr()), ctypes.c_void_p(ov_d.data_ptr()),
        ctypes.c_void_p(stream.cuda_stream))
    torch.cuda.synchronize(dev)
    return st, dens_d.cpu().numpy().copy(), float(ov_d.item())


def _check(torch, nl, chip, with_half):
    dev = torch.device("cuda:0")
    torch.cuda.set_device(dev)
    half_d = None
    if with_half:
        half = np.stack([nl.cell_w.astype(np.float32) * 0.5, nl.cell_h.astype(np.float32) * 0.5], axis=1)
        half_d = torch.from_numpy(np.ascontiguousarray(half)).to(dev)
    dens_d = torch.full((chip.bins_y or chip.height, chip.bins_x or chip.width), -1.0, dtype=torch.float64,
                        device=dev)
    ov_d = torch.full((1,), -1.0, dtype=torch.float64, device=dev)
    orc = Oracle(nl, chip)
    with E.PlacementContext(nl, chip) as ctx:
        for call, seed in enumerate((31, 32)):
            x, y = _positions(nl, chip, seed)
            ref_d, ref_ov = ctx.density(x, y)
            st, got, ov = _noalloc(torch, nl, chip, x, y, half_d, dens_d, ov_d)
            assert st == _abi.EPLACE_OK, (call, st)
            assert np.array_equal(got, ref_d), call
            assert abs(ov - ref_ov) <= 1e-12 * max(1.0, abs(ref_ov)), call
            od = orc.density(x, y)
            assert rel_err(got, od) <= 1e-5, call
            assert abs(ov - orc.overlap(od)) <= 1e-6, call


def test_density_noalloc_with_footprints():
    """Macros of 2..8 sites and two sites per bin edge."""
    import torch

    nl, chip = E.synth_netlist(E.SynthSpec(seed=5, num_cells=12000, num_nets=13200, num_pads=600, width=256,
                                           height=256, bins_x=128, bins_y=128, cluster_size=64,
                                           macro_fraction=0.05))
    _check(torch, nl, chip, with_half=True)


def test_density_noalloc_unit_cells():
    """All cells 1x1 and half_wh = NULL: the unit-cell path of the scatter."""
    import torch

    nl, chip = E.synth_netlist(E.SynthSpec(seed=6, num_cells=9000, num_nets=9900, num_pads=300, width=160,
                                           height=120, cluster_size=32))
    assert nl.cell_w is None
    _check(torch, nl, chip, with_half=False)


def test_density_noalloc_empty_design():
    """No cells: a zero map and overlap 0, also right after a call that
    filled the working array."""
    import torch

    dev = torch.device("cuda:0")
    torch.cuda.set_device(dev)
    full, chip = E.synth_netlist(E.SynthSpec(seed=7, num_cells=3000, num_nets=3300, num_pads=100, width=64,
                                             height=64, cluster_size=32))
    empty = E.Netlist(num_cells=0, net_offsets=np.zeros(1, np.uint32), pin_cell=np.zeros(0, np.uint32))
    dens_d = torch.full((64, 64), -1.0, dtype=torch.float64, device=dev)
    ov_d = torch.full((1,), -1.0, dtype=torch.float64, device=dev)
    x, y = _positions(full, chip, 3)
    st, got, _ = _noalloc(torch, full, chip, x, y, None, dens_d, ov_d)
    assert st == _abi.EPLACE_OK and got.sum() > 0
    e = np.zeros(0, np.float32)
    st, got, ov = _noalloc(torch, empty, chip, e, e, None, dens_d, ov_d)
    assert st == _abi.EPLACE_OK
    assert not got.any() and ov == 0.0


def test_density_noalloc_rejects_bad_arguments():
    """Rejected on the host, before anything reaches the device: a grid above
    the 512 x 512 working array, and device pointers that are not 8-byte
    aligned."""
    import torch

    L = _abi.lib()
    st = L.eplace_density_noalloc(None, None, 0, 1024, 1024, 1024, 1024, ctypes.c_void_p(8), ctypes.c_void_p(8),
                                  None)
    assert st == _abi.EPLACE_ERR_INVALID
    dev = torch.device("cuda:0")
    buf = torch.zeros(4096, dtype=torch.float64, device=dev)
    base = buf.data_ptr()
    assert base % 256 == 0
    for pos, half, dens, ov in ((base + 4, 0, base + 2048, base + 3072),
                                (base, base + 4, base + 2048, base + 3072),
                                (base, 0, base + 2052, base + 3072),
                                (base, 0, base + 2048, base + 3076)):
        st = L.eplace_density_noalloc(ctypes.c_void_p(pos), ctypes.c_void_p(half), 8, 64, 64, 16, 16,
                                      ctypes.c_void_p(dens), ctypes.c_void_p(ov), None)
        assert st == _abi.EPLACE_ERR_INVALID, (pos - base, half, dens - base, ov - base)


@pytest.mark.parametrize("cells,w,h,bx,by", [(1, 7, 5, 7, 5), (31, 33, 17, 33, 17), (33, 64, 64, 16, 8),
                                             (257, 90, 60, 45, 30), (4099, 512, 256, 512, 256)])
@pytest.mark.parametrize("half", ["unit", "mixed"])
def test_density_noalloc_shapes(cells, w, h, bx, by, half):
    """Counts of cells and bins around a warp and around the four-bin groups,
    footprints within and beyond 2 x 2 bins (0.5 to 6 bins wide, any half
    extent), some of them partly outside the chip: against the overlaps in
    FP64, bins within 1e-6 of the largest (a bin is a sum of FP32 areas, each
    exact to 2^-23, rounded to 2^-32), the overlap within 1e-6."""
    import torch

    dev = torch.device("cuda:0")
    torch.cuda.set_device(dev)
    rng = np.random.default_rng(cells)
    nl = E.Netlist(num_cells=cells, net_offsets=np.zeros(1, np.uint32), pin_cell=np.zeros(0, np.uint32))
    chip = E.Chip(w, h, bx, by)
    x, y = rng.uniform(-1, w, cells).astype(np.float32), rng.uniform(-1, h, cells).astype(np.float32)
    hf = np.full((cells, 2), 0.5, np.float32)
    if half == "mixed":
        hf = np.where(rng.random((cells, 1)) < 0.3, rng.uniform(0.25, 3.0 * w / bx, (cells, 2)), hf).astype(np.float32)
    half_d = torch.from_numpy(hf).to(dev) if half == "mixed" else None
    dens_d = torch.full((by, bx), -1.0, dtype=torch.float64, device=dev)
    ov_d = torch.full((1,), -1.0, dtype=torch.float64, device=dev)
    sx, sy = w // bx, h // by

    def axis(c, e, s, n):  # [cells, n] lengths in the bins
        lo, hi = c.astype(np.float64) - e, c.astype(np.float64) + e
        k = np.arange(n)
        return np.maximum(np.minimum(hi[:, None], (k + 1) * s) - np.maximum(lo[:, None], k * s), 0.0)

    want = axis(y, hf[:, 1], sy, by).T @ axis(x, hf[:, 0], sx, bx)
    over = np.maximum(want - sx * sy, 0).sum() / want.sum()
    for _ in range(2):  # the second call finds the scratch as the first left it
        st, got, ov = _noalloc(torch, nl, chip, x, y, half_d, dens_d, ov_d)
        assert st == _abi.EPLACE_OK
        assert np.abs(got - want).max() <= 1e-6 * want.max()
        assert abs(ov - over) <= 1e-6


def _axis(c, e, s, n):  # [cells, n] lengths of [c - e, c + e] in n bins of s sites
    lo, hi = c.astype(np.float64) - e, c.astype(np.float64) + e
    k = np.arange(n)
    return np.maximum(np.minimum(hi[:, None], (k + 1) * s) - np.maximum(lo[:, None], k * s), 0.0)


@pytest.mark.parametrize("cells,side,bins,extent", [
    (200, 4096, 512, 2000.0),     # 2^31 sites and more of footprints in all, a bin far below
    (900, 4096, 512, 2000.0),     # 2^32 and more
    (3, 16384, 1, 8192.0),        # one bin of 2^28 sites, three times over
    (5, 46341, 1, 700.0),         # bins of 2^31 sites and of 2^32: cells fill little of them
    (5, 65536, 1, 700.0),
    (5, 131072, 2, 700.0),
])
def test_density_noalloc_large_areas(cells, side, bins, extent):
    """Areas beyond 2^31 sites, in all bins together or as a bin's capacity:
    bins and overlap within 1e-6 as for small ones."""
    import torch

    dev = torch.device("cuda:0")
    torch.cuda.set_device(dev)
    rng = np.random.default_rng(cells)
    nl = E.Netlist(num_cells=cells, net_offsets=np.zeros(1, np.uint32), pin_cell=np.zeros(0, np.uint32))
    chip = E.Chip(side, side, bins, bins)
    x, y = rng.uniform(0.45 * side, 0.55 * side, (2, cells)).astype(np.float32)
    hf = np.full((cells, 2), extent, np.float32)
    half_d = torch.from_numpy(hf).to(dev)
    dens_d = torch.full((bins, bins), -1.0, dtype=torch.float64, device=dev)
    ov_d = torch.full((1,), -1.0, dtype=torch.float64, device=dev)
    s = side // bins
    want = _axis(y, hf[:, 1], s, bins).T @ _axis(x, hf[:, 0], s, bins)
    over = np.maximum(want - float(s) * s, 0).sum() / want.sum()
    assert want.max() < 2.0 ** 31  # what a bin holds
    st, got, ov = _noalloc(torch, nl, chip, x, y, half_d, dens_d, ov_d)
    assert st == _abi.EPLACE_OK
    assert np.abs(got - want).max() <= 1e-6 * want.max()
    assert abs(ov - over) <= 1e-6


def test_density_stage_large_areas():
    """The same through the regular density entry: 60,000 macros of 255 x 255
    sites, 3.4e9 sites of footprints in all."""
    n, side, bins = 60000, 4096, 256
    rng = np.random.default_rng(1)
    w = np.full(n, 255, np.uint8)
    nl = E.Netlist(num_cells=n, net_offsets=np.zeros(1, np.uint32), pin_cell=np.zeros(0, np.uint32), cell_w=w, cell_h=w)
    x, y = rng.uniform(0.1 * side, 0.9 * side, (2, n)).astype(np.float32)
    half = np.full(n, 127.5)
    s = side // bins
    want = _axis(y, half, s, bins).T @ _axis(x, half, s, bins)
    over = np.maximum(want - float(s) * s, 0).sum() / want.sum()
    with E.PlacementContext(nl, E.Chip(side, side, bins, bins)) as ctx:
        got, ov = ctx.density(x, y)
    assert np.abs(got - want).max() <= 1e-6 * want.max()
    assert abs(ov - over) <= 1e-6


def test_density_noalloc_after_overlapping_calls():
    """Calls that overlap on the GPU spoil each other's results, but no later
    call's: the next ones are right, map and overlap."""
    import torch

    L = _abi.lib()
    dev = torch.device("cuda:0")
    torch.cuda.set_device(dev)
    torch.cuda.synchronize(dev)
    rng = np.random.default_rng(4)
    streams = [torch.cuda.Stream(dev) for _ in range(3)]
    work = []
    for k, (cells, side, bins) in enumerate(((150000, 1024, 512), (2000, 128, 64), (0, 96, 96))):
        nl = E.Netlist(num_cells=cells, net_offsets=np.zeros(1, np.uint32), pin_cell=np.zeros(0, np.uint32))
        x, y = rng.uniform(0, side - 1, (2, cells)).astype(np.float32)
        pos = torch.from_numpy(np.ascontiguousarray(np.stack([x, y], axis=1))).to(dev)
        work.append((nl, E.Chip(side, side, bins, bins), x, y, pos,
                     torch.zeros((bins, bins), dtype=torch.float64, device=dev),
                     torch.zeros(1, dtype=torch.float64, device=dev)))
    torch.cuda.synchronize(dev)
    for _ in range(3):
        for _ in range(200):
            for s, (nl, chip, x, y, pos, dens, ov) in zip(streams, work):
                st = L.eplace_density_noalloc(
                    ctypes.c_void_p(pos.data_ptr() if nl.num_cells else 0), None, nl.num_cells, chip.width, chip.height,
                    chip.bins_x, chip.bins_y, ctypes.c_void_p(dens.data_ptr()), ctypes.c_void_p(ov.data_ptr()),
                    ctypes.c_void_p(s.cuda_stream))
                assert st == _abi.EPLACE_OK
        torch.cuda.synchronize(dev)
        for nl, chip, x, y, pos, dens, ov in work:
            ov.fill_(-1.0)
            with E.PlacementContext(nl, chip) as ctx:
                want, ref = ctx.density(x, y)
            st, got, o = _noalloc(torch, nl, chip, x, y, None, dens, ov)
            assert st == _abi.EPLACE_OK
            assert np.array_equal(got, want) and abs(o - ref) <= 1e-12


@pytest.mark.parametrize("cells", [1, 33, 700])
@pytest.mark.parametrize("share,bins_wide", [(1.0, 1.0), (1.0, 5.0), (0.05, 1.0), (0.05, 9.0), (0.5, 2.5)])
def test_density_noalloc_shares_of_wide_footprints(cells, share, bins_wide):
    """Warps in which all, half and few cells cover more than 2 x 2 bins, up to
    a bin or two more than a warp has lanes."""
    import torch

    dev = torch.device("cuda:0")
    torch.cuda.set_device(dev)
    rng = np.random.default_rng(cells)
    nl = E.Netlist(num_cells=cells, net_offsets=np.zeros(1, np.uint32), pin_cell=np.zeros(0, np.uint32))
    w, h, bx, by = 240, 160, 60, 80  # 4 x 2 sites a bin
    chip = E.Chip(w, h, bx, by)
    x, y = rng.uniform(0, w - 1, cells).astype(np.float32), rng.uniform(0, h - 1, cells).astype(np.float32)
    wide = rng.random(cells) < share
    hf = np.where(wide[:, None], np.array([[2.0 * bins_wide, 1.0 * bins_wide]]), 0.5).astype(np.float32)
    dens_d = torch.full((by, bx), -1.0, dtype=torch.float64, device=dev)
    ov_d = torch.full((1,), -1.0, dtype=torch.float64, device=dev)
    want = _axis(y, hf[:, 1], 2, by).T @ _axis(x, hf[:, 0], 4, bx)
    over = np.maximum(want - 8.0, 0).sum() / want.sum()
    st, got, ov = _noalloc(torch, nl, chip, x, y, torch.from_numpy(hf).to(dev), dens_d, ov_d)
    assert st == _abi.EPLACE_OK
    assert np.abs(got - want).max() <= 1e-6 * want.max()
    assert abs(ov - over) <= 1e-6
