"""The step's shares of the cells: counts around a warp and a block, designs of
macros only (more macro tasks than warps), footprints of more bins than the
eight columns and five rows a group of lanes takes at once; the gather and one
whole step against the oracle with the tolerances of the parity tests, and a
short run in one cooperative launch per step against the same run in the job
engine, which takes the step as three launches."""

import numpy as np
import pytest

import eisenjoch_b200 as E
from oracle.oracle import Oracle
from tests.conftest import rel_err

pytestmark = pytest.mark.gpu


def design(n, macros, side, seed):
    rng = np.random.default_rng(seed)
    cw = np.ones(n, np.uint8)
    ch = np.ones(n, np.uint8)
    m = {"none": np.zeros(n, bool), "some": rng.random(n) < 0.3, "all": np.ones(n, bool)}[macros]
    cw[m], ch[m] = rng.integers(1, 20, m.sum()), rng.integers(1, 20, m.sum())
    nets = max(1, n // 2)
    pins = rng.integers(0, n, 2 * nets).astype(np.uint32)
    nl = E.Netlist(num_cells=n, net_offsets=np.arange(0, 2 * nets + 1, 2, dtype=np.uint32), pin_cell=pins,
                   cell_w=cw, cell_h=ch)
    return nl, E.Chip(side, side)


@pytest.mark.parametrize("n", [1, 31, 33, 129, 2049])
@pytest.mark.parametrize("macros", ["none", "some", "all"])
def test_gather_and_step_shares(n, macros):
    nl, chip = design(n, macros, 96, 7 * n + len(macros))
    rng = np.random.default_rng(n)
    orc = Oracle(nl, chip)
    W, H = chip.width, chip.height
    ex, ey = rng.normal(0, 1, (2, H, W)).astype(np.float32)
    x, y = rng.uniform(0, W - 1, n).astype(np.float32), rng.uniform(0, H - 1, n).astype(np.float32)
    xp, yp = np.clip(x + 0.3, 0, W - 1).astype(np.float32), np.clip(y - 0.3, 0, H - 1).astype(np.float32)
    gw = rng.normal(0, 0.3, (2, n)).astype(np.float32)
    gp = rng.normal(0, 0.05, (2, n)).astype(np.float32)
    with E.PlacementContext(nl, chip) as ctx:
        gx, gy = ctx.gather(x, y, ex, ey)
        ox, oy = orc.gather(x, y, ex, ey)
        assert rel_err(gx, ox) <= 1e-5 and rel_err(gy, oy) <= 1e-5
        for it, lam in ((0, 0.0), (5, 2.5)):
            state = dict(x=x, y=y, x_prev=xp, y_prev=yp, gprev_x=gp[0], gprev_y=gp[1])
            scal = [lam, float(lam > 0), 0.1, 0.2]
            nx, ny, ax, ay, lx, ly = ctx.step(it, x, y, gw[0], gw[1], ex, ey, state, scal)
            ref, norms = orc.step(it, dict(x=x, y=y, x_prev=xp, y_prev=yp, gprev_x=gp[0], gprev_y=gp[1], step_x=0.1,
                                           step_y=0.2, density_penalty=lam, initialized=lam > 0), gw[0], gw[1], ox, oy)
            # the penalty's start is a quotient of two norms of FP32 gradients
            assert abs(scal[0] - ref["density_penalty"]) <= 1e-5 * max(1.0, abs(ref["density_penalty"]))
            assert abs(ax - ref["step_x"]) <= 1e-4 * ref["step_x"] and abs(ay - ref["step_y"]) <= 1e-4 * ref["step_y"]
            for k in ("x", "y", "x_prev", "y_prev"):
                assert np.abs(state[k] - ref[k]).max() <= 2e-4 + 1e-5 * np.abs(ref[k]).max(), k
            assert abs(nx - norms[0]) <= 1e-4 * norms[0] + 1e-6 and abs(ny - norms[1]) <= 1e-4 * norms[1] + 1e-6
            assert np.abs(lx - ref["look_x"]).max() <= 1e-3 and np.abs(ly - ref["look_y"]).max() <= 1e-3


@pytest.mark.parametrize("n", [33, 700, 21000])
def test_step_in_one_launch_and_in_three(n):
    """(21,000 cells: blocks of 256 threads.)"""
    spec = E.SynthSpec(seed=n, num_cells=n, num_nets=n, num_pads=40, width=256, height=256, bins_x=128, bins_y=64,
                       cluster_size=32, macro_fraction=0.04)
    nl, chip = E.synth_netlist(spec)
    cfg = E.ElectroPlaceCfg(max_iters=23, legalize_interval=4)
    opts = E.RunOptions(field_mode=1)
    with E.PlacementContext(nl, chip) as ctx:
        a = ctx.run(cfg, opts)
    with E.JobServer(max_jobs=1, opts=opts) as srv:
        b, _ = srv.wait(srv.submit(nl, chip, cfg))
    assert np.array_equal(a.x, b.x) and np.array_equal(a.y, b.y) and np.array_equal(a.bel_tile, b.bel_tile)
    assert a.trajectory == b.trajectory


@pytest.mark.parametrize("n,side,bins,macros", [(100, 32, 16, 0.0), (1000, 64, 64, 0.05), (5000, 128, 128, 0.05),
                                                (21000, 256, 64, 0.0)])
@pytest.mark.parametrize("it", [16, 30])
def test_scatter_of_cells_piled_up_in_a_bin(n, side, bins, macros, it):
    """The reference's field drives the cells to the edges and into the
    corners.  The density that step `it` scatters (lanes of one bin add
    together) against the density entry point's (each cell adds its own) at
    the same look-ahead, by the overlap of the next checkpoint: sums of whole
    numbers on both sides, a few FP64 operations after them."""
    nl, chip = E.synth_netlist(E.SynthSpec(seed=n, num_cells=n, num_nets=n, num_pads=40, width=side, height=side,
                                           bins_x=bins, bins_y=bins, cluster_size=32, macro_fraction=macros))
    opts = E.RunOptions(field_mode=0)
    with E.PlacementContext(nl, chip) as ctx:
        before, now, after = (ctx.run(E.ElectroPlaceCfg(max_iters=k + 1, legalize_interval=k), opts)
                              for k in (it - 1, it, it + 1))
        assert before.best_iter == it - 1 and now.best_iter == it
        a = [1.0]
        while len(a) < it + 3:
            a.append((1 + np.sqrt(1 + 4 * a[-1] ** 2)) / 2)
        m = (a[it + 1] - 1) / a[it + 2]

        def look(p, q):
            p, q = p.astype(np.float64), q.astype(np.float64)
            return np.clip((p + m * (p - q)).astype(np.float32), 0, np.float32(side - 1))

        d, ov = ctx.density(look(now.x, before.x), look(now.y, before.y))
    got = next(t["overlap"] for t in after.trajectory if t["iter"] == it + 1)
    assert abs(got - ov) <= 1e-12


@pytest.mark.parametrize("it,lam", [(0, 0.0), (0, 2.5), (5, 2.5)])
def test_entries_on_an_empty_design(it, lam):
    """No movable cell: every stage entry takes it, and reads no cell."""
    nl = E.Netlist(num_cells=0, net_offsets=np.array([0, 2], np.uint32), pin_cell=np.array([0, 1], np.uint32),
                   fixed_x=np.array([3, 20], np.int32), fixed_y=np.array([5, 9], np.int32))
    chip = E.Chip(32, 32)
    z = np.zeros(0, np.float32)
    rng = np.random.default_rng(0)
    ex, ey = rng.normal(0, 1, (2, 32, 32)).astype(np.float32)
    with E.PlacementContext(nl, chip) as ctx:
        state = {k: z for k in ("x", "y", "x_prev", "y_prev", "gprev_x", "gprev_y")}
        scal = [lam, float(lam > 0), 0.1, 0.2]
        nx, ny, ax, ay, lx, ly = ctx.step(it, z, z, z, z, ex, ey, state, scal)
        assert nx == 0.0 and ny == 0.0 and ax == 0.1 and ay == 0.2 and len(lx) == len(ly) == 0
        gx, gy = ctx.gather(z, z, ex, ey)
        wx, wy = ctx.wa_grad(z, z)
        assert len(gx) == len(gy) == len(wx) == len(wy) == 0
        d, ov = ctx.density(z, z)
        assert not d.any() and ov == 0.0
        sx, sy, disp, _ = ctx.legalize_device(z, z)
        assert len(sx) == len(sy) == 0 and disp == 0.0
