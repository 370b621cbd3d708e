"""The device legaliser against the host legaliser and the oracle's
brute-force scan: identical bindings, identical FP64 displacement (bit for
bit) and the identical integer HPWL, on uniform, piled, tied (k + 1/2),
off-grid and over-full inputs, with and without macros, with the free map in
shared memory and in global memory; and whole runs with the device
legaliser equal to runs with the host legaliser."""

import numpy as np
import pytest

import eisenjoch_b200 as E
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu

CASES = {
    "unit_128": E.SynthSpec(seed=1, num_cells=5000, num_nets=5500, num_pads=400, width=128, height=128,
                            bins_x=128, bins_y=128, cluster_size=32),
    "macro_256_bins128": E.SynthSpec(seed=5, num_cells=12000, num_nets=13200, num_pads=600, width=256, height=256,
                                     bins_x=128, bins_y=128, cluster_size=64, macro_fraction=0.05),
    "odd_90x60": E.SynthSpec(seed=7, num_cells=1500, num_nets=1650, num_pads=100, width=90, height=60,
                             cluster_size=32),
    # 1280 x 1280: the free map (215 KB) lives in global memory
    "global_map_1280": E.SynthSpec(seed=8, num_cells=40000, num_nets=44000, num_pads=800, width=1280, height=1280,
                                   bins_x=256, bins_y=256, cluster_size=64, macro_fraction=0.02),
}


@pytest.fixture(scope="module", params=sorted(CASES))
def case(request):
    nl, chip = E.synth_netlist(CASES[request.param])
    ctx = E.PlacementContext(nl, chip)
    yield request.param, nl, chip, ctx
    ctx.close()


def layouts(nl, chip, seed):
    """Uniform, piled (a few tight clusters: long searches), and positions
    on half-integers (ties between two or four nearest sites)."""
    rng = np.random.default_rng(seed)
    n, W, H = nl.num_cells, chip.width, chip.height
    out = {}
    out["uniform"] = (rng.uniform(0, W - 1, n), rng.uniform(0, H - 1, n))
    k = rng.integers(0, 4, n)
    cx, cy = rng.uniform(0.2, 0.8, 4) * (W - 1), rng.uniform(0.2, 0.8, 4) * (H - 1)
    out["piled"] = (cx[k] + rng.normal(0, W * 0.01, n), cy[k] + rng.normal(0, H * 0.01, n))
    out["half"] = (np.floor(rng.uniform(0, W - 1, n)) + 0.5 * rng.integers(0, 2, n),
                   np.floor(rng.uniform(0, H - 1, n)) + 0.5 * rng.integers(0, 2, n))
    res = {}
    for name, (x, y) in out.items():
        res[name] = (np.clip(x, 0, W - 1).astype(np.float32), np.clip(y, 0, H - 1).astype(np.float32))
    return res


def test_device_legalizer_matches_host(case):
    name, nl, chip, ctx = case
    for lname, (x, y) in layouts(nl, chip, 23).items():
        hx, hy, hd = ctx.legalize(x, y)
        dx, dy, dd, dh = ctx.legalize_device(x, y)
        assert np.array_equal(dx, hx) and np.array_equal(dy, hy), (name, lname)
        assert dd == hd, (name, lname, dd, hd)
        assert dh == E.hpwl_host(nl, chip, hx, hy), (name, lname)


def test_device_legalizer_matches_oracle_scan():
    """Against the oracle's exhaustive scan (the reference's loop as written)."""
    nl, chip = E.synth_netlist(CASES["odd_90x60"])
    ctx = E.PlacementContext(nl, chip)
    orc = Oracle(nl, chip)
    try:
        for lname, (x, y) in layouts(nl, chip, 31).items():
            dx, dy, dd, dh = ctx.legalize_device(x, y)
            st, ox, oy, od = orc.legalize(x, y, 0)
            assert st == 0
            assert np.array_equal(dx, ox) and np.array_equal(dy, oy), lname
            assert dd == od, lname
            assert dh == orc.hpwl(dx, dy)
    finally:
        ctx.close()


def test_device_legalizer_off_grid_positions():
    """Unclamped inputs (outside [0, W-1]) skip the nearest-point shortcut
    and are searched from the clamped row, as on the host."""
    nl, chip = E.synth_netlist(CASES["odd_90x60"])
    ctx = E.PlacementContext(nl, chip)
    try:
        rng = np.random.default_rng(5)
        n = nl.num_cells
        x = rng.uniform(-20, chip.width + 20, n).astype(np.float32)
        y = rng.uniform(-20, chip.height + 20, n).astype(np.float32)
        hx, hy, hd = ctx.legalize(x, y)
        dx, dy, dd, _ = ctx.legalize_device(x, y)
        assert np.array_equal(dx, hx) and np.array_equal(dy, hy)
        assert dd == hd
    finally:
        ctx.close()


def test_device_legalizer_full_chip():
    """Exactly as many cells as sites: every site is used; one more cell
    than sites: NoBelsAvailable, as on the host."""
    W = H = 24
    n = W * H
    nl = E.Netlist(num_cells=n, net_offsets=np.array([0, 2], np.uint32), pin_cell=np.array([0, 1], np.uint32))
    chip = E.Chip(W, H)
    ctx = E.PlacementContext(nl, chip)
    try:
        rng = np.random.default_rng(9)
        x = np.full(n, 11.3, np.float32) + rng.normal(0, 1, n).astype(np.float32)
        y = np.full(n, 12.6, np.float32) + rng.normal(0, 1, n).astype(np.float32)
        hx, hy, hd = ctx.legalize(x, y)
        dx, dy, dd, _ = ctx.legalize_device(x, y)
        assert np.array_equal(dx, hx) and np.array_equal(dy, hy) and dd == hd
        assert len(np.unique(dy * W + dx)) == n
    finally:
        ctx.close()
    nl2 = E.Netlist(num_cells=n + 1, net_offsets=np.array([0, 2], np.uint32), pin_cell=np.array([0, 1], np.uint32))
    ctx2 = E.PlacementContext(nl2, chip)
    try:
        x = np.full(n + 1, 3.0, np.float32)
        with pytest.raises(E.NoBelsAvailable):
            ctx2.legalize(x, x)
        with pytest.raises(E.NoBelsAvailable):
            ctx2.legalize_device(x, x)
    finally:
        ctx2.close()


@pytest.mark.parametrize("field_mode", [1, 0])
def test_run_with_device_legalizer_equals_host(field_mode):
    nl, chip, cfg = E.workload("electro_5k_128")
    if field_mode == 0:
        cfg.max_iters = 60
    a = E.place_electro(nl, chip, cfg, E.RunOptions(field_mode=field_mode, legal_mode=0))
    b = E.place_electro(nl, chip, cfg, E.RunOptions(field_mode=field_mode, legal_mode=1))
    assert a.hpwl == b.hpwl and a.best_iter == b.best_iter and a.iters == b.iters
    assert np.array_equal(a.bel_tile, b.bel_tile)
    assert np.array_equal(a.x, b.x) and np.array_equal(a.y, b.y)
    assert a.trajectory == b.trajectory


def test_run_with_device_legalizer_macros():
    nl, chip = E.synth_netlist(CASES["macro_256_bins128"])
    cfg = E.ElectroPlaceCfg(max_iters=80)
    a = E.place_electro(nl, chip, cfg, E.RunOptions(field_mode=1, legal_mode=0))
    b = E.place_electro(nl, chip, cfg, E.RunOptions(field_mode=1, legal_mode=1))
    assert a.hpwl == b.hpwl and a.best_iter == b.best_iter
    assert np.array_equal(a.bel_tile, b.bel_tile)
    assert a.trajectory == b.trajectory


def test_device_legalizer_bench_geometry():
    """The benchmark job's geometry (200k cells, 5 % macros, 1024^2 sites)
    with the cells drawn into one central pile, as in the crowded middle of
    a run (many cells end up ~200 sites from their target, in long chains
    of cells that depend on each other): the device legaliser's bindings,
    displacement and HPWL equal the host legaliser's bit for bit."""
    nl, chip, _ = E.workload("electro_200k_1024")
    rng = np.random.default_rng(41)
    n, W = nl.num_cells, chip.width
    x = np.clip(rng.normal(W / 2, W * 0.13, n), 0, W - 1).astype(np.float32)
    y = np.clip(rng.normal(W / 2, W * 0.13, n), 0, W - 1).astype(np.float32)
    with E.PlacementContext(nl, chip) as ctx:
        hx, hy, hd = ctx.legalize(x, y)
        dx, dy, dd, dh = ctx.legalize_device(x, y)
    assert np.array_equal(dx, hx) and np.array_equal(dy, hy)
    assert dd == hd
    assert dh == E.hpwl_host(nl, chip, hx, hy)


@pytest.mark.parametrize("w,h", [(31, 40), (32, 33), (33, 32), (64, 64), (70, 45), (257, 40)])
@pytest.mark.parametrize("macros", ["none", "small", "large"])
def test_device_legalizer_edges(w, h, macros):
    """Chips whose width is no multiple of the 32-site segments, blocked
    sites, and footprints on either side of what the word search takes
    (32 x 16 sites): all cells on one spot, on two corners, and uniform."""
    rng = np.random.default_rng(w * 100 + h)
    sizes = {"none": [(1, 1)] * 8, "small": [(2, 2), (8, 8), (3, 5), (1, 9), (12, 1)],
             "large": [(32, 16), (31, 17), (16, 30), (1, 31), (31, 1)]}[macros]
    cw, ch, area = [], [], 0
    for k in range(4 if macros == "large" else 24):
        a, b = sizes[k % len(sizes)]
        if a <= w and b <= h and area + 3 * a * b < w * h // 2:
            cw.append(a)
            ch.append(b)
            area += 3 * a * b  # room for the blocks that fragments cost
    units = (w * h - area) // 2
    cw, ch = np.array(cw + [1] * units, np.uint8), np.array(ch + [1] * units, np.uint8)
    n = len(cw)
    perm = rng.permutation(n)
    cw, ch = cw[perm], ch[perm]
    fx, fy = rng.integers(0, w, 5).astype(np.int32), rng.integers(0, h, 5).astype(np.int32)
    nl = E.Netlist(num_cells=n, net_offsets=np.array([0, 2], np.uint32), pin_cell=np.array([0, 1], np.uint32),
                   fixed_x=fx, fixed_y=fy, fixed_on_logic=np.ones(5, np.uint8), cell_w=cw, cell_h=ch)
    chip = E.Chip(w, h)
    corner = rng.random(n) < 0.5
    spots = [(np.full(n, 0.37 * w), np.full(n, 0.61 * h)),
             (np.where(corner, 0.0, w - 1.0), np.where(corner, 0.0, h - 1.0)),
             (rng.uniform(0, w - 1, n), rng.uniform(0, h - 1, n))]
    with E.PlacementContext(nl, chip) as ctx:
        for x, y in spots:
            try:
                hx, hy, hd = ctx.legalize(x, y)
            except E.NoBelsAvailable:
                with pytest.raises(E.NoBelsAvailable):
                    ctx.legalize_device(x, y)
                continue
            dx, dy, dd, dh = ctx.legalize_device(x, y)
            assert np.array_equal(dx, hx) and np.array_equal(dy, hy)
            assert dd == hd
            assert dh == E.hpwl_host(nl, chip, hx, hy)


@pytest.mark.parametrize("n,side", [(16383, 256), (16384, 256), (17408, 256), (17409, 140), (16900, 130)])
@pytest.mark.parametrize("macros", [0, 12])
def test_device_legalizer_all_at_once(n, side, macros):
    """Unit cells that are placed all at once and those left over: counts
    around where that starts and around the chunks they are listed by, from
    hardly any left over to all of them, on an open and on a full chip."""
    rng = np.random.default_rng(n + macros)
    cw = np.ones(n, np.uint8)
    cw[rng.permutation(n)[:macros]] = 4  # 4 x 1
    if n + 3 * macros > side * side:
        n -= 3 * macros
        cw = np.sort(cw)[::-1][:n].copy()
    nl = E.Netlist(num_cells=n, net_offsets=np.array([0, 2], np.uint32), pin_cell=np.array([0, 1], np.uint32),
                   cell_w=cw, cell_h=np.ones(n, np.uint8))
    chip = E.Chip(side, side)
    grid = np.arange(n) * (side * side // n)
    own_site = np.stack([grid % side, grid // side]).astype(np.float64)
    uniform = rng.uniform(0, side - 1, (2, n))
    with E.PlacementContext(nl, chip) as ctx:
        for piled in (0.0, 0.05, 0.12, 1.0):
            p = own_site if piled == 0.0 else uniform.copy()
            m = rng.random(n) < piled
            p = np.where(m, side * 0.4 + rng.normal(0, side * 0.02, (2, n)), p)
            x, y = np.clip(p, 0, side - 1).astype(np.float32)
            hx, hy, hd = ctx.legalize(x, y)
            dx, dy, dd, _ = ctx.legalize_device(x, y)
            assert np.array_equal(dx, hx) and np.array_equal(dy, hy), piled
            assert dd == hd


@pytest.mark.parametrize("field_mode", [0, 1])
def test_run_with_device_legalizer_all_at_once(field_mode):
    """A run long enough to legalise checkpoints that are no longer wanted."""
    nl, chip = E.synth_netlist(E.SynthSpec(seed=11, num_cells=24000, num_nets=26000, num_pads=200, width=256,
                                           height=256, bins_x=128, bins_y=128, cluster_size=64, macro_fraction=0.02))
    cfg = E.ElectroPlaceCfg(max_iters=60)
    a = E.place_electro(nl, chip, cfg, E.RunOptions(field_mode=field_mode, legal_mode=0))
    for _ in range(2):
        b = E.place_electro(nl, chip, cfg, E.RunOptions(field_mode=field_mode, legal_mode=1))
        assert a.hpwl == b.hpwl and a.best_iter == b.best_iter
        assert np.array_equal(a.bel_tile, b.bel_tile)
        assert a.trajectory == b.trajectory


@pytest.mark.parametrize("macros", [False, True])
@pytest.mark.parametrize("far", [1e2, 1e4, 1e6, 1.1e7])
def test_device_legalizer_targets_off_the_chip(far, macros):
    """Targets beside, above and diagonally off the chip, some of them one on
    another (the displaced cells' lists), up to 2^24 sites away."""
    rng = np.random.default_rng(int(far))
    n, w, h = 300, 70, 40
    cw = np.ones(n, np.uint8)
    if macros:
        cw[rng.permutation(n)[:20]] = 3
    nl = E.Netlist(num_cells=n, net_offsets=np.array([0, 2], np.uint32), pin_cell=np.array([0, 1], np.uint32),
                   cell_w=cw, cell_h=cw if macros else None)
    with E.PlacementContext(nl, E.Chip(w, h)) as ctx:
        for dx, dy in ((1, 0), (-1, 0), (0, 1), (0, -1), (1, 1), (-1, 0.3)):
            x, y = rng.uniform(0, w - 1, n), rng.uniform(0, h - 1, n)
            off = rng.random(n) < 0.5
            x, y = np.where(off, 0.4 * w + dx * far, x), np.where(off, 0.6 * h + dy * far, y)
            hx, hy, hd = ctx.legalize(x, y)
            gx, gy, gd, _ = ctx.legalize_device(x, y)
            assert np.array_equal(gx, hx) and np.array_equal(gy, hy)
            assert gd == hd


@pytest.mark.parametrize("cells", [40, 16384])
@pytest.mark.parametrize("bad", [(2.0 ** 25, 5.0), (5.0, -(2.0 ** 25)), (1e19, 5.0), (5.0, 2e19), (-3e38, 3e38),
                                 (np.inf, 5.0), (5.0, -np.inf), (np.nan, 5.0), (5.0, np.nan)])
def test_device_legalizer_refuses_targets_without_a_site(cells, bad):
    """A target that is no number, infinite or too far away (FP32 costs of its
    sites are infinite from 2^64 sites on): the call ends with an error, and the
    next one is right."""
    side = 8 if cells == 40 else 160
    rng = np.random.default_rng(cells)
    nl = E.Netlist(num_cells=cells, net_offsets=np.array([0, 2], np.uint32), pin_cell=np.array([0, 1], np.uint32))
    x, y = rng.uniform(0, side - 1, (2, cells)).astype(np.float32)
    with E.PlacementContext(nl, E.Chip(side, side)) as ctx:
        for which in (0, cells // 2, cells - 1):
            fx, fy = x.copy(), y.copy()
            fx[which], fy[which] = bad
            with pytest.raises(E.NoBelsAvailable):
                ctx.legalize_device(fx, fy)
        hx, hy, hd = ctx.legalize(x, y)
        gx, gy, gd, _ = ctx.legalize_device(x, y)
        assert np.array_equal(gx, hx) and np.array_equal(gy, hy) and gd == hd


@pytest.mark.parametrize("n,piles", [(3000, 1), (15000, 3), (30000, 1), (30000, 8)])
def test_device_legalizer_long_chains(n, piles):
    """Piles whose cells displace one another in long chains, each displaced
    cell going by the list that another CTA wrote: the same binding every time."""
    rng = np.random.default_rng(n + piles)
    side = 256
    nl = E.Netlist(num_cells=n, net_offsets=np.array([0, 2], np.uint32), pin_cell=np.array([0, 1], np.uint32))
    k = rng.integers(0, piles, n)
    c = rng.uniform(0.3 * side, 0.7 * side, (2, piles))
    x, y = np.clip(c[:, k] + rng.normal(0, 1.5, (2, n)), 0, side - 1).astype(np.float32)
    with E.PlacementContext(nl, E.Chip(side, side)) as ctx:
        hx, hy, hd = ctx.legalize(x, y)
        for _ in range(3):
            gx, gy, gd, _ = ctx.legalize_device(x, y)
            assert np.array_equal(gx, hx) and np.array_equal(gy, hy) and gd == hd


@pytest.mark.parametrize("n", [40, 255, 256, 257, 700, 5000, 16383, 16384, 17000])
@pytest.mark.parametrize("macros", [0, 9])
def test_device_legalizer_cells_on_one_target(n, macros):
    """Many cells on one target, alone and beside others, in corners, on edges,
    nearly equal, off the chip, and around the counts from which cells are
    placed in windows and all at once; blocked sites around the target."""
    rng = np.random.default_rng(n + macros)
    side = 32 if n < 800 else 96 if n <= 5000 else 140
    cw = np.ones(n, np.uint8)
    cw[rng.permutation(n)[:macros]] = 3
    fx, fy = rng.integers(0, side // 2, (2, 20)).astype(np.int32)
    nl = E.Netlist(num_cells=n, net_offsets=np.array([0, 2], np.uint32), pin_cell=np.array([0, 1], np.uint32),
                   fixed_x=fx, fixed_y=fy, fixed_on_logic=np.ones(20, np.uint8), cell_w=cw, cell_h=np.ones(n, np.uint8))
    u = rng.uniform(0, side - 1, (2, n))
    spread = lambda share, x, y: np.where(rng.random(n) < share, np.array([[x], [y]]), u)
    k = rng.integers(0, 3, n)
    spots = rng.uniform(0.2 * side, 0.8 * side, (2, 3))
    layouts = {
        "spot": np.array([[0.37 * side], [0.61 * side]]) + np.zeros((2, n)),
        "half": np.full((2, n), side // 2 + 0.5),  # four sites tie
        "corner": spread(0.97, 0.0, 0.0),
        "corner, others": spread(0.4, side - 1.0, 0.0),
        "few": spread(0.04, 0.0, side - 1.0),
        "spots": spots[:, k],
        "nearly": np.array([[0.4 * side], [0.5 * side]]) + rng.normal(0, 0.004, (2, n)),
        "in a pile": np.where(rng.random(n) < 0.5, 0.5 * side, 0.5 * side + rng.normal(0, 0.06 * side, (2, n))),
        "off": spread(0.8, -300.0, 0.3 * side),
    }
    with E.PlacementContext(nl, E.Chip(side, side)) as ctx:
        for name, (x, y) in layouts.items():
            hx, hy, hd = ctx.legalize(x, y)
            for _ in range(2):
                gx, gy, gd, _ = ctx.legalize_device(x, y)
                assert np.array_equal(gx, hx) and np.array_equal(gy, hy), name
                assert gd == hd, name


@pytest.mark.parametrize("side", [16, 130])
def test_device_legalizer_full_chip_on_one_target(side):
    """As many cells as sites, all on one target, and one more than that."""
    for n, fits in ((side * side, True), (side * side + 1, False)):
        nl = E.Netlist(num_cells=n, net_offsets=np.array([0, 2], np.uint32), pin_cell=np.array([0, 1], np.uint32))
        x = np.full(n, 0.25 * side, np.float32)
        try:
            ctx = E.PlacementContext(nl, E.Chip(side, side))
        except E.NoBelsAvailable:
            assert not fits
            continue
        with ctx:
            if not fits:
                with pytest.raises(E.NoBelsAvailable):
                    ctx.legalize_device(x, x)
                continue
            hx, hy, hd = ctx.legalize(x, x)
            gx, gy, gd, _ = ctx.legalize_device(x, x)
            assert np.array_equal(gx, hx) and np.array_equal(gy, hy) and gd == hd


@pytest.mark.parametrize("cells,side,bins", [(1000, 64, 64), (20000, 200, 100)])
def test_run_with_device_legalizer_and_reference_field(cells, side, bins):
    """The reference's field leaves most cells on one corner: the same run as
    with the host legaliser, checkpoints no longer wanted among them."""
    nl, chip = E.synth_netlist(E.SynthSpec(seed=5, num_cells=cells, num_nets=cells, num_pads=60, width=side,
                                           height=side, bins_x=bins, bins_y=bins, cluster_size=32))
    cfg = E.ElectroPlaceCfg(max_iters=70)
    a = E.place_electro(nl, chip, cfg, E.RunOptions(legal_mode=0))
    b = E.place_electro(nl, chip, cfg, E.RunOptions(legal_mode=1))
    assert a.hpwl == b.hpwl and np.array_equal(a.bel_tile, b.bel_tile) and a.trajectory == b.trajectory


@pytest.mark.parametrize("w,h", [(32, 17), (33, 1), (33, 33), (40, 40), (63, 31), (64, 32), (65, 3), (96, 34), (97, 64),
                                 (130, 65), (1, 100)])
@pytest.mark.parametrize("blocked", [0, 25])
def test_device_legalizer_large_macros(w, h, blocked):
    """Footprints beyond what the word search takes, around multiples of 32 along
    both axes, on one spot, spread, and beside blocked sites: against the
    oracle's exhaustive scan."""
    rng = np.random.default_rng(w * 1000 + h + blocked)
    W, H, macros, units = 300, 170, 4, 150
    cw, ch = np.ones(macros + units, np.uint8), np.ones(macros + units, np.uint8)
    cw[:macros], ch[:macros] = [w, w, max(w - 1, 1), w], [h, max(h - 1, 1), h, h]
    fx, fy = rng.integers(0, W, blocked).astype(np.int32), rng.integers(0, H, blocked).astype(np.int32)
    nl = E.Netlist(num_cells=macros + units, net_offsets=np.array([0, 2], np.uint32),
                   pin_cell=np.array([0, 1], np.uint32), fixed_x=fx, fixed_y=fy,
                   fixed_on_logic=np.ones(blocked, np.uint8), cell_w=cw, cell_h=ch)
    chip = E.Chip(W, H)
    orc = Oracle(nl, chip)
    n = macros + units
    with E.PlacementContext(nl, chip) as ctx:
        for x, y in ((np.full(n, 0.47 * W), np.full(n, 0.53 * H)), (np.zeros(n), np.full(n, H - 1.0)),
                     (rng.uniform(0, W - 1, n), rng.uniform(0, H - 1, n))):
            st, ox, oy, od = orc.legalize(x.astype(np.float32), y.astype(np.float32), 0)
            if st != 0:
                with pytest.raises(E.NoBelsAvailable):
                    ctx.legalize_device(x, y)
                continue
            gx, gy, gd, _ = ctx.legalize_device(x, y)
            assert np.array_equal(gx, ox) and np.array_equal(gy, oy)
            assert gd == od
