"""The work that a user of this placer has it do, as timed cases.

Whole placements (one-shot, on a resident netlist, with the legaliser on the
device, a batch through the job engine) and the layers of the iteration that a
program can call by themselves (density, wirelength gradient, field solve,
fused step, legaliser).  Sizes are those of the benchmark workloads
(5,000 / 200,000 cells, 128^2 to 1024^2 bins), of the mixed-size job streams
(1k cells and up, 64^2 bins and up) and of the parity tests (grids that are
not powers of two), and `draw` spreads over the ranges between them.
"""

import ctypes

import numpy as np
import torch

import eisenjoch_b200 as E
from eisenjoch_b200 import _abi

POTENTIAL_GRADIENT = _abi.EPLACE_FIELD_POTENTIAL_GRADIENT


# ---------------------------------------------------------------------------
# The cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # A control loop that asks for the density of a small design on device
        # buffers of its own: a call of a few microseconds, where launches count.
        dict(name="density_dev_2k_64", kind="density", cells=2000, macros=0.0, site=128, bin=64),
        # The same call at the largest grid it takes, with macro footprints.
        dict(name="density_dev_200k_512", kind="density", cells=200000, macros=0.05, site=1024, bin=512),
        # The wirelength gradient alone, as another analytical placer uses it,
        # at the 200k-cell benchmark netlist.
        dict(name="wa_200k", kind="wa", cells=200000, macros=0.05, site=1024, bin=512),
        # One fused gather / penalty / Barzilai-Borwein / FISTA step of the
        # same netlist, on state that the caller holds.
        dict(name="step_200k_512", kind="step", cells=200000, macros=0.05, site=1024, bin=512, iter=30),
        # The field of a density map: the default transform at the benchmark grid.
        dict(name="field_fft_512", kind="field", cells=2000, bx=512, by=512, per=2, mode="fft", gradient=True),
        # The mixed-precision transform at the grid of the 800k-cell workload.
        dict(name="field_tc_1024", kind="field", cells=2000, bx=1024, by=1024, per=2, mode="tc", gradient=True),
        # A grid that is no power of two (the matrix form), reference formula.
        dict(name="field_gemm_200x120", kind="field", cells=2000, bx=200, by=120, per=1, mode="fft", gradient=False),
        # Legalising one checkpoint of the 200k-cell job on the device.
        dict(name="legal_dev_200k", kind="legal", cells=200000, macros=0.05, site=1024, bin=512),
        # The smallest benchmark workload with the default options: 300
        # iterations of the reference's field formula on a resident netlist.
        dict(name="run_5k_128_reference", kind="run", cells=5000, macros=0.0, site=128, bin=128, gradient=False,
             iters=300, legal="host", mode="fft", oneshot=False),
        # A medium job that leaves no work to the host cores (device legaliser).
        dict(name="run_30k_256_device", kind="run", cells=30000, macros=0.05, site=512, bin=256, gradient=True,
             iters=500, legal="gpu", mode="fft", oneshot=False),
        # The headline: one 200k-cell netlist from host buffers to bindings.
        dict(name="place_200k_512", kind="run", cells=200000, macros=0.05, site=1024, bin=512, gradient=True,
             iters=500, legal="host", mode="fft", oneshot=True),
        # A service's batch: twelve mixed jobs through the job engine.
        dict(name="engine_12_jobs", kind="engine", jobs=12, low=2000, high=40000),
    ]


def _log(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["density", "wa", "step", "field", "legal", "run", "run", "engine"])
    if kind == "field":
        mode = rng.choice(["fft", "fft", "tc", "simt"])
        if mode == "tc":
            bx, by = 64 * rng.randint(1, 8), 128 * rng.randint(1, 4)
        elif mode == "fft":
            bx, by = 2 ** rng.randint(4, 10), 2 ** rng.randint(4, 10)
        else:  # any grid; sides that are and are not multiples of 8
            bx, by = _log(rng, 20, 300), _log(rng, 20, 300)
        return dict(kind=kind, cells=rng.randint(500, 4000), bx=bx, by=by, per=rng.choice([1, 2]), mode=mode,
                    gradient=rng.random() < 0.5)
    if kind == "engine":
        low = _log(rng, 1000, 4000)
        return dict(kind=kind, jobs=rng.randint(2, 12), low=low, high=_log(rng, 8000, 40000))
    # netlists of 1k to 200k cells; the bin grid as the mixed job streams pick
    # it, at times a grid that is no power of two, at times one site per bin
    cells = _log(rng, 1000, 200000)
    b = 64
    while b * b < cells and b < 512:
        b *= 2
    if kind != "density" and rng.random() < 0.25:
        b = b + rng.randint(1, 24)
    if kind == "density" and b < 512:
        b = b + rng.randint(0, 40)
    per = 1 if b * b > 2.2 * cells and rng.random() < 0.3 else 2
    macros = rng.choice([0.0, 0.05]) if per == 2 else 0.0
    case = dict(kind=kind, cells=cells, macros=macros, site=per * b, bin=b)
    if kind == "step":
        case["iter"] = rng.choice([0, 1, 30])
    if kind == "run":
        gradient = rng.random() < 0.75
        case.update(gradient=gradient, iters=120 if gradient else 60,
                    legal="gpu" if cells <= 40000 and rng.random() < 0.3 else "host",
                    mode="tc" if b % 128 == 0 and rng.random() < 0.3 else "fft", oneshot=rng.random() < 0.5)
    return case


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
def _netlist(case, seed):
    n = case["cells"]
    spec = E.SynthSpec(seed=seed * 1000 + n, num_cells=n, num_nets=int(round(1.1 * n)), num_pads=max(40, n // 100),
                       width=case["site"], height=case["site"], bins_x=case["bin"], bins_y=case["bin"],
                       cluster_size=64, macro_fraction=case["macros"])
    return E.synth_netlist(spec)


def _positions(nl, chip, seed):
    """Cells on the way to being spread: half of them anywhere, half in six piles."""
    rng = np.random.default_rng([seed, 1])
    n, w, h = nl.num_cells, chip.width, chip.height
    cx, cy = rng.uniform(0.3, 0.7, 6) * (w - 1), rng.uniform(0.3, 0.7, 6) * (h - 1)
    k = rng.integers(0, 6, n)
    pile = rng.random(n) < 0.5
    x = np.where(pile, cx[k] + rng.normal(0, 0.06 * w, n), rng.uniform(0.05, 0.95, n) * (w - 1))
    y = np.where(pile, cy[k] + rng.normal(0, 0.06 * h, n), rng.uniform(0.05, 0.95, n) * (h - 1))
    return np.clip(x, 0, w - 1).astype(np.float32), np.clip(y, 0, h - 1).astype(np.float32)


def _half(nl):
    if nl.cell_w is None:
        return np.full((nl.num_cells, 2), 0.5, np.float32)
    return np.stack([0.5 * nl.cell_w, 0.5 * nl.cell_h], axis=1).astype(np.float32)


def _smooth(bx, by, seed):
    """A map of long waves, as a field or the uneven part of a density has."""
    rng = np.random.default_rng([seed, 2])
    fx, fy = np.arange(bx) / bx, np.arange(by) / by
    m = np.zeros((by, bx))
    for _ in range(6):
        a, b, p, q = rng.uniform(0, 12), rng.uniform(0, 12), rng.uniform(0, 6), rng.uniform(0, 6)
        m += rng.uniform(0.1, 1) * np.outer(np.cos(b * fy + p), np.cos(a * fx + q))
    return m


def _step_inputs(case, nl, chip, seed):
    rng = np.random.default_rng([seed, 3])
    n, w, h = nl.num_cells, chip.width, chip.height
    x, y = _positions(nl, chip, seed)
    f = lambda v, top: np.clip(v, 0, top).astype(np.float32)  # noqa: E731
    xp, yp = f(x + rng.normal(0, 0.3, n), w - 1), f(y + rng.normal(0, 0.3, n), h - 1)
    if case["iter"] == 0:
        xp, yp = x.copy(), y.copy()
    m = _momentum(case["iter"] + 2)[case["iter"]]
    lx, ly = f(x + m * (x.astype(np.float64) - xp), w - 1), f(y + m * (y.astype(np.float64) - yp), h - 1)
    g = rng.normal(0, 0.4, (4, n)).astype(np.float32)
    ex = _smooth(case["bin"], case["bin"], seed + 10).astype(np.float32)
    ey = _smooth(case["bin"], case["bin"], seed + 20).astype(np.float32)
    first = case["iter"] == 0
    state = dict(x=x, y=y, x_prev=xp, y_prev=yp, gprev_x=0.1 * g[2] * (not first), gprev_y=0.1 * g[3] * (not first))
    state = {k: np.ascontiguousarray(v, np.float32) for k, v in state.items()}
    return dict(look=(lx, ly), gwl=(g[0], g[1]), field=(ex, ey), state=state,
                scal=[0.0 if first else 3.7, 0.0 if first else 1.0, 0.1, 0.1 if first else 0.2])


def _job_specs(case, seed):
    """The stream's sizes are the case's own, its netlists the seed's."""
    return E.placer.mixed_job_specs(case["jobs"], 1000 * seed + 1, case["low"], case["high"], rng_seed=case["jobs"])


_DCT = {"fft": _abi.EPLACE_DCT_FP32_FFT, "tc": _abi.EPLACE_DCT_BF16X3_TC, "simt": _abi.EPLACE_DCT_FP32_SIMT}


def prepare(case, seed):
    kind = case["kind"]
    if kind == "engine":
        jobs = [E.synth_netlist(s) for s in _job_specs(case, seed)]
        opts = E.RunOptions(field_mode=POTENTIAL_GRADIENT, dct_mode=_abi.EPLACE_DCT_BF16X3_TC)
        return dict(case=case, jobs=jobs, server=E.JobServer(max_jobs=case["jobs"], opts=opts))
    if kind == "field":
        per = case["per"]
        spec = E.SynthSpec(seed=seed, num_cells=min(case["cells"], case["bx"] * case["by"] * per * per // 2),
                           num_nets=case["cells"], num_pads=40, width=per * case["bx"], height=per * case["by"],
                           bins_x=case["bx"], bins_y=case["by"])
        nl, chip = E.synth_netlist(spec)
        rng = np.random.default_rng([seed, 4])
        d = 0.5 + 0.2 * _smooth(case["bx"], case["by"], seed) + rng.exponential(0.3, (case["by"], case["bx"]))
        return dict(case=case, ctx=E.PlacementContext(nl, chip), density=np.maximum(d, 0.0))
    nl, chip = _netlist(case, seed)
    if kind == "run":
        cfg = E.ElectroPlaceCfg(seed=seed + 1, max_iters=case["iters"])
        opts = E.RunOptions(field_mode=POTENTIAL_GRADIENT if case["gradient"] else _abi.EPLACE_FIELD_REFERENCE,
                            dct_mode=_DCT[case["mode"]],
                            legal_mode=_abi.EPLACE_LEGAL_GPU if case["legal"] == "gpu" else _abi.EPLACE_LEGAL_HOST)
        s = dict(case=case, nl=nl, chip=chip, cfg=cfg, opts=opts)
        if not case["oneshot"]:
            s["ctx"] = E.PlacementContext(nl, chip)
        return s
    if kind == "step":
        return dict(case=case, ctx=E.PlacementContext(nl, chip), **_step_inputs(case, nl, chip, seed))
    x, y = _positions(nl, chip, seed)
    if kind == "density":
        dev = torch.device("cuda")
        b = case["bin"]
        return dict(case=case, n=nl.num_cells, fn=_abi.lib().eplace_density_noalloc,
                    pos=torch.from_numpy(np.stack([x, y], axis=1)).to(dev),
                    half=torch.from_numpy(_half(nl)).to(dev) if case["macros"] else None,
                    density=torch.zeros((b, b), dtype=torch.float64, device=dev),
                    overlap=torch.zeros(1, dtype=torch.float64, device=dev))
    return dict(case=case, ctx=E.PlacementContext(nl, chip), x=x, y=y)  # wa, legal


# ---------------------------------------------------------------------------
# One pass
# ---------------------------------------------------------------------------
def _placement(r):
    return dict(x=r.x, y=r.y, bel_tile=r.bel_tile, hpwl=r.hpwl, iters=r.iters)


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "density":
        b, w = case["bin"], case["site"]
        st = s["fn"](ctypes.c_void_p(s["pos"].data_ptr()),
                     ctypes.c_void_p(s["half"].data_ptr() if s["half"] is not None else 0), s["n"], w, w, b, b,
                     ctypes.c_void_p(s["density"].data_ptr()), ctypes.c_void_p(s["overlap"].data_ptr()),
                     ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        if st != _abi.EPLACE_OK:
            raise RuntimeError("eplace_density_noalloc: status %d" % st)
        return s["density"], s["overlap"]
    if kind == "wa":
        return s["ctx"].wa_grad(s["x"], s["y"])
    if kind == "step":
        state, scal = dict(s["state"]), list(s["scal"])
        nx, ny, ax, ay, lx, ly = s["ctx"].step(case["iter"], *s["look"], *s["gwl"], *s["field"], state, scal)
        return dict(state=state, look_x=lx, look_y=ly, scalars=np.array([scal[0], scal[2], scal[3], ax, ay, nx, ny]))
    if kind == "field":
        return s["ctx"].field(s["density"], dct_mode=_DCT[case["mode"]],
                              field_mode=POTENTIAL_GRADIENT if case["gradient"] else _abi.EPLACE_FIELD_REFERENCE)
    if kind == "legal":
        return s["ctx"].legalize_device(s["x"], s["y"])
    if kind == "engine":
        ids = [s["server"].submit(nl, chip, E.ElectroPlaceCfg()) for nl, chip in s["jobs"]]
        return [_placement(s["server"].wait(i)[0]) for i in ids]
    if case["oneshot"]:
        return _placement(E.place_electro(s["nl"], s["chip"], s["cfg"], s["opts"]))
    return _placement(s["ctx"].run(s["cfg"], s["opts"]))


# ---------------------------------------------------------------------------
# What a pass cannot do without
# ---------------------------------------------------------------------------
PINS_PER_NET = 7.1  # of the netlist generator, duplicates dropped


def _iteration(cells, bins):
    """Bytes and operations of one iteration: the netlist and positions of the
    wirelength gradient, the density map, the field, the solver's state."""
    pins = PINS_PER_NET * 1.1 * cells
    wa = 4 * 1.1 * cells + 4 * pins + 16 * cells
    density = 8 * cells + 8 * bins
    field = 12 * bins
    step = 68 * cells + 8 * bins
    return wa + density + field + step, 60 * pins + 30 * bins * max(1.0, np.log2(max(bins, 2))) + 100 * cells


def work(case):
    kind = case["kind"]
    if kind == "field":
        bins = case["bx"] * case["by"]
        return dict(bytes=16 * bins, flops=15 * bins * np.log2(bins))
    if kind == "engine":  # the fewest iterations the stopping rule allows are 21
        n = case["jobs"] * (case["high"] - case["low"]) / np.log(case["high"] / case["low"])
        b, f = _iteration(n, n)
        return dict(bytes=21 * b, flops=21 * f)
    n, bins = case["cells"], case["bin"] ** 2
    pins = PINS_PER_NET * 1.1 * n
    if kind == "density":
        return dict(bytes=8 * n + (8 * n if case["macros"] else 0) + 8 * bins + 8, flops=30 * n)
    if kind == "wa":
        return dict(bytes=4.4 * n + 4 * pins + 16 * n, flops=60 * pins)
    if kind == "step":
        return dict(bytes=88 * n + 8 * bins, flops=100 * n)
    if kind == "legal":
        return dict(bytes=16 * n + case["site"] ** 2 / 8 + 4.4 * n + 4 * pins, flops=20 * n)
    b, f = _iteration(n, bins)
    iters = 21 if case["gradient"] else case["iters"]
    return dict(bytes=iters * b, flops=iters * f)


# ---------------------------------------------------------------------------
# The layers' results in 64 bits
# ---------------------------------------------------------------------------
def _overlaps(p, h, s, bins):
    """First bin and the lengths of [p - h, p + h] in the bins from there on."""
    lo, hi = p - h, p + h
    b0 = np.clip(np.floor(lo / s).astype(np.int64), 0, bins)
    most = int((np.ceil(hi / s) - b0).max())
    b = b0[:, None] + np.arange(most)
    o = np.minimum(hi[:, None], (b + 1) * s) - np.maximum(lo[:, None], b * s)
    return b, np.where(b < bins, np.maximum(o, 0.0), 0.0)


def _footprints(nl, chip, x, y, bin_):
    half = _half(nl).astype(np.float64)
    bx, ox = _overlaps(x.astype(np.float64), half[:, 0], chip.width // bin_, bin_)
    by, oy = _overlaps(y.astype(np.float64), half[:, 1], chip.height // bin_, bin_)
    return np.minimum(bx, bin_ - 1), ox, np.minimum(by, bin_ - 1), oy


def _exact_density(case, seed):
    nl, chip = _netlist(case, seed)
    x, y = _positions(nl, chip, seed)
    b = case["bin"]
    bx, ox, by, oy = _footprints(nl, chip, x, y, b)
    d = np.zeros(b * b)
    for i in range(bx.shape[1]):
        for j in range(by.shape[1]):
            d += np.bincount(by[:, j] * b + bx[:, i], ox[:, i] * oy[:, j], b * b)
    cap = float((case["site"] // b) ** 2)
    return d.reshape(b, b), np.array([np.maximum(d - cap, 0).sum() / d.sum()])


def _exact_wa(case, seed):
    nl, chip = _netlist(case, seed)
    x, y = _positions(nl, chip, seed)
    off = nl.net_offsets.astype(np.int64)
    deg = np.diff(off)
    pins, n, gamma = nl.pin_cell.astype(np.int64), nl.num_cells, 0.5
    used = np.repeat(deg >= 2, deg)
    out = []
    for pos, fixed in ((x, nl.fixed_x), (y, nl.fixed_y)):
        p = np.concatenate([pos.astype(np.float64), fixed.astype(np.float64)])[pins]
        seg = off[:-1][deg > 0]
        at = np.cumsum(deg > 0)[np.repeat(np.arange(len(deg)), deg)] - 1
        u, v = p - np.maximum.reduceat(p, seg)[at], p - np.minimum.reduceat(p, seg)[at]
        ep, em = np.exp(gamma * u), np.exp(-gamma * v)
        total = lambda q: np.add.reduceat(q, seg)[at]  # noqa: E731
        sp, sm = total(ep), total(em)
        g = ep / sp * (1 + gamma * (u - total(u * ep) / sp)) - em / sm * (1 - gamma * (v - total(v * em) / sm))
        move = used & (pins < n)
        out.append(np.bincount(pins[move], g[move], n))
    return tuple(out)


def _exact_field(case, seed):
    bx, by, per = case["bx"], case["by"], case["per"]
    n = min(case["cells"], bx * by * per * per // 2)
    rng = np.random.default_rng([seed, 4])
    d = np.maximum(0.5 + 0.2 * _smooth(bx, by, seed) + rng.exponential(0.3, (by, bx)), 0.0)
    rho = d - n / (bx * by)

    def tables(m):
        k, t = np.arange(m), (np.arange(m) + 0.5) / m
        dct2 = np.cos(np.pi * np.outer(k, t))
        cos3 = dct2.T * np.where(k == 0, 0.5, 1.0)
        if case["gradient"]:
            sin3 = -np.sin(np.pi * np.outer(t, k))
        else:
            sin3 = np.sin(np.pi * np.outer(t, k + 1)) * np.where(k == m - 1, 0.5, 1.0)
        return dct2, cos3, sin3, np.pi * k / m

    cx, c3x, s3x, wx = tables(bx)
    cy, c3y, s3y, wy = tables(by)
    a = cy @ rho @ cx.T * (4.0 / (bx * by))
    a[0, :] *= 0.5
    a[:, 0] *= 0.5
    den = 2 * (1 - np.cos(wx))[None, :] + 2 * (1 - np.cos(wy))[:, None]
    den[0, 0] = 1.0
    a[0, 0] = 0.0
    phi = a / den
    return c3y @ (phi * wx[None, :]) @ s3x.T, s3y @ (phi * wy[:, None]) @ c3x.T


def _momentum(n):
    m, a = [], 1.0
    for _ in range(n):
        nxt = (1 + np.sqrt(1 + 4 * a * a)) / 2
        m.append((a - 1) / nxt)
        a = nxt
    return m


def _exact_step(case, seed):
    nl, chip = _netlist(case, seed)
    s = _step_inputs(case, nl, chip, seed)
    it, b, n = case["iter"], case["bin"], nl.num_cells
    half = _half(nl).astype(np.float64)
    area = 4 * half[:, 0] * half[:, 1]
    bx, ox, by, oy = _footprints(nl, chip, *s["look"], b)
    fx, fy, wt = np.zeros(n), np.zeros(n), np.zeros(n)
    for i in range(bx.shape[1]):
        for j in range(by.shape[1]):
            w = ox[:, i] * oy[:, j]
            fx += w * s["field"][0][by[:, j], bx[:, i]].astype(np.float64)
            fy += w * s["field"][1][by[:, j], bx[:, i]].astype(np.float64)
            wt += w
    den = np.stack([area * fx / wt, area * fy / wt])
    gwl = np.stack(s["gwl"]).astype(np.float64)
    lam, init = s["scal"][0], s["scal"][1]
    if init:
        lam = lam * 1.025 if lam < 50 else lam + 1
    else:
        lam = 0.1 * np.linalg.norm(gwl) / np.linalg.norm(den)
    deg = np.diff(nl.net_offsets.astype(np.int64))
    pins = nl.pin_cell.astype(np.int64)
    w = np.repeat(np.where(deg >= 2, 1.0 / np.maximum(deg, 1), 0.0), deg)
    pw = np.bincount(pins[pins < n], w[pins < n], n)
    g = (gwl + lam * den) / np.maximum(pw + lam * area, 1.0)
    st = {k: v.astype(np.float64) for k, v in s["state"].items()}
    x, xp = np.stack([st["x"], st["y"]]), np.stack([st["x_prev"], st["y_prev"]])
    gp = np.stack([st["gprev_x"], st["gprev_y"]])
    alpha = np.array(s["scal"][2:4])
    if it > 0:
        dx, dg = x - xp, g - gp
        alpha = np.clip(np.abs((dx * dx).sum(1) / (dx * dg).sum(1)), 1e-4, 1.0)
    m = _momentum(it + 2)
    new = x + m[it] * (x - xp) - alpha[:, None] * g
    norm = np.sqrt(((new - x) ** 2).sum(1))
    top = np.array([[chip.width - 1.0], [chip.height - 1.0]])
    new, old = np.clip(new, 0, top), np.clip(x, 0, top)
    look = np.clip(new + m[it + 1] * (new - old), 0, top)
    state = dict(x=new[0], y=new[1], x_prev=old[0], y_prev=old[1], gprev_x=g[0], gprev_y=g[1])
    return dict(state=state, look_x=look[0], look_y=look[1],
                scalars=np.array([lam, alpha[0], alpha[1], alpha[0], alpha[1], norm[0], norm[1]]))


def exact(case, seed):
    """Whole placements and legalisations have none: they end in whole numbers."""
    of = {"density": _exact_density, "wa": _exact_wa, "field": _exact_field, "step": _exact_step}.get(case["kind"])
    return of(case, seed) if of else None
