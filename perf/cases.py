"""The work that users of the solver have it do, as cases that can be timed.

A case is one pass through the public entry points (the C ABI and its Python
host) from what a program has in hand: a built case, a handle with the state
resident on the device, host buffers in pinned memory for what it reads back.

  flow      outer iterations of the resident state, then the state read back,
            as a run that saves its fields does (Sphase.f90:37-235, Sav3f.f90)
  start     the same from host fields: upload and INITSV in every pass
  batch     outer iterations of several furnaces in flight together
  radiation the volume radiation transfer on the band model and the wall
            exchange after it (RAD_EMIS)
  emission  the emission-only radiation update (rad_qe_only)
  msflow    minor species and soot on the frozen flow (MSFLOW)
  adlbl3    one line solve of a host system (CALL ADLBL3)
  learned   a training step of the learned p' start: forward, gradients, Adam

Grids: the synthetic furnaces of gfm_gb300.configs (48x24x16 to 192x96x64,
the batched variants' ranges, odd extents among them) and the reference's own
cases in tests/golden with their restarts.  Precision: FP64 and mixed; plane
order: the reference's march and the red-black order.

Furnaces start from their fresh start with a through-flow (a guess that a
user sets, or a coarser run's state): seeded smooth modes on a plug flow with
the inlets' jets and developed k and eps.  The fresh start at rest amplifies rounding a
thousandfold per iteration, so two builds could not be compared on it.

The mixed path holds its fields in FP32 on the device; the pass converts
what comes back to FP32 (exactly), as a program that keeps such a state does.
"""
from __future__ import annotations

import ctypes as C
import dataclasses
import lzma
import math
import pathlib
import random
import shutil
import tempfile

import numpy as np
import torch

from gfm_gb300 import Case, GpuSolver, abi, configs
from gfm_gb300.lp import LearnedPressure
from gfm_gb300.solver import Fields, gflow_batch

ROOT = pathlib.Path(__file__).resolve().parent.parent
GOLD = ROOT / "tests" / "golden"
ADI = {"march": abi.GFM_ADI_MARCH, "redblack": abi.GFM_ADI_REDBLACK}
PREC = {"fp64": abi.GFM_PREC_FP64, "mixed": abi.GFM_PREC_MIXED}
STATE = ("p", "t", "ug", "gf")      # what a restart or a plot of the gas state takes


# ---- the cases ---------------------------------------------------------------

def listed() -> list:
    return [
        # What a user of the reference gets with the defaults: a shipped case
        # from its files and restart, FP64, the reference's plane order.
        {"name": "tc21_march_fp64", "kind": "flow", "grid": "0041", "prec": "fp64", "adi": "march", "iters": 2},
        # The same case in the production order and mixed precision: small
        # planes, where latency and the number of launches count.
        {"name": "tc21_mixed", "kind": "flow", "grid": "0041", "prec": "mixed", "adi": "redblack", "iters": 5},
        # The longer end-fired furnace, FP64 with the red-black order.
        {"name": "endfired_fp64", "kind": "flow", "grid": "1207", "prec": "fp64", "adi": "redblack", "iters": 4},
        # A furnace of odd extents from host fields: a parameter study's step.
        {"name": "start_ragged_mixed", "kind": "start", "grid": "87x45x29", "prec": "mixed", "adi": "redblack", "iters": 8},
        # The benchmark furnace, mixed precision: the production run.
        {"name": "furnace_mixed", "kind": "flow", "grid": "192x96x64", "prec": "mixed", "adi": "redblack", "iters": 20},
        # The benchmark furnace in plain FP64.
        {"name": "furnace_fp64", "kind": "flow", "grid": "192x96x64", "prec": "fp64", "adi": "redblack", "iters": 4},
        # A parameter study: furnace variants in flight together.
        {"name": "batch_mixed", "kind": "batch", "variants": 8, "set": 7, "prec": "mixed", "iters": 4},
        # A full radiation call of the shipped case: band model, volume
        # transfer, wall exchange.
        {"name": "radiation_tc21", "kind": "radiation", "grid": "0041", "prec": "fp64"},
        # The emission update inside an iteration series, benchmark furnace.
        {"name": "emission_mixed", "kind": "emission", "grid": "192x96x64", "prec": "mixed"},
        # Minor species between radiation calls, shipped case.
        {"name": "msflow_tc21", "kind": "msflow", "grid": "0041", "prec": "fp64", "iters": 10},
        # A Fortran host that replaces CALL ADLBL3 alone.
        {"name": "adlbl3_fp64", "kind": "adlbl3", "grid": "96x48x32", "prec": "fp64", "adi": "redblack", "sweeps": 6},
        # The learned p' start in training, on the grid it is trained on.
        {"name": "learned_train", "kind": "learned", "grid": "48x24x16"},
    ]


def _extent(rng: random.Random, lo: int, hi: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _grid(rng: random.Random, nx=(24, 192), ny=(14, 96), nz=(10, 64)) -> str:
    return "%dx%dx%d" % (_extent(rng, *nx), _extent(rng, *ny), _extent(rng, *nz))


def draw(rng: random.Random) -> dict:
    kind = rng.choice(["flow"] * 5 + ["start", "batch", "radiation", "emission", "msflow", "adlbl3", "learned"])
    prec = rng.choice(["fp64", "mixed"])
    real = rng.choice(["0041", "1207"])
    if kind in ("flow", "start"):
        adi = rng.choice(["redblack"] * 4 + ["march"])
        if adi == "march":   # the plane order walks every plane: small grids
            grid = rng.choice([real, _grid(rng, (12, 32), (8, 20), (6, 16))])
            iters = rng.randint(1, 2)
        else:
            grid = real if kind == "flow" and rng.random() < 0.25 else _grid(rng)
            iters = rng.randint(1, 4) if prec == "fp64" else rng.randint(2, 12)
        if grid in ("0041", "1207"):
            iters = min(iters, 5)
        return {"kind": kind, "grid": grid, "prec": prec, "adi": adi, "iters": iters}
    if kind == "batch":
        return {"kind": kind, "variants": rng.randint(2, 12), "set": rng.randint(8, 10 ** 4), "prec": prec, "iters": rng.randint(1, 4)}
    if kind == "radiation":
        return {"kind": kind, "grid": _grid(rng, (10, 32), (8, 16), (6, 12)), "prec": "fp64"}
    if kind == "emission":
        return {"kind": kind, "grid": _grid(rng), "prec": prec}
    if kind == "msflow":
        return {"kind": kind, "grid": real, "prec": "fp64", "iters": rng.randint(2, 11)}
    if kind == "adlbl3":
        return {"kind": kind, "grid": _grid(rng, (24, 128), (14, 64), (10, 48)), "prec": prec,
                "adi": "redblack", "sweeps": rng.randint(1, 8)}
    even = [2 * (_extent(rng, lo, hi) // 2) for lo, hi in ((16, 128), (12, 64), (8, 48))]
    return {"kind": kind, "grid": "%dx%dx%d" % tuple(even)}


# ---- states ------------------------------------------------------------------

class State:
    """What the program keeps between passes."""

    def __init__(self, **kw):
        self.__dict__.update(kw)


def _modes(rng, shape, n=4, kmax=3):
    """A smooth field of unit size on the unit box: n seeded cosine products."""
    ax = [np.linspace(0.0, 1.0, m) for m in shape]
    out = np.zeros(shape)
    for _ in range(n):
        f = [np.cos(math.pi * rng.integers(1, kmax + 1) * a + rng.uniform(0.0, 2.0 * math.pi)) for a in ax]
        out += f[0][:, None, None] * f[1][None, :, None] * f[2][None, None, :]
    return out / n


# A start-up run's factors: heavy relaxation while the flow establishes itself,
# and no wall sink, which the reference turns on with its first radiation call
# (the shipped cases here have it on).  With the furnace's own factors a change
# of rounding grows to the size of the fields within ten iterations.
RUN = {"rf_uvw": 0.1, "rfl_h": 0.1, "rfl_k": 0.1, "rfl_eps": 0.1, "rfl_species": 0.1, "rf_hsource": 0.1, "wall_sink": 0}


def _furnace(grid: str, seed: int) -> Case:
    nx, ny, nz = (int(v) for v in grid.split("x"))
    return Case(configs.furnace_variant(seed % 100003, nx, ny, nz, aspect=2.0, **RUN))


def _shipped(num: str, minor: bool = False, **kw):
    """A shipped case from its files and its end-of-run restarts."""
    gold = GOLD / f"case{num}"
    with tempfile.TemporaryDirectory() as d:
        d = pathlib.Path(d)
        for f in gold.iterdir():
            if f.is_file() and f.suffix == ".xz":
                (d / f.stem).write_bytes(lzma.decompress(f.read_bytes()))
            elif f.is_file():
                shutil.copyfile(f, d / f.name)
        case = Case.from_files(d, num, restart=True, **kw)
        return case, (case.read_minor(d / f"rs{num}c.d") if minor else None)


def _through_flow(case: Case, rng) -> Fields:
    """The fresh start with a seeded through-flow, the inlets' jets reaching
    into the furnace, and developed turbulence."""
    f = case.initial_fields()
    ib = case.ibcell()
    op = ib <= 0
    a = f.arrays
    shape = op.shape
    w = np.sin(math.pi * np.linspace(0, 1, shape[1]))[None, :, None] * np.sin(math.pi * np.linspace(0, 1, shape[0]))[:, None, None]
    jet = np.where(ib == 2, a["ug"][0], 0.0).max(axis=2)[:, :, None] * np.exp(-0.5 * np.linspace(0, 1, shape[2]))
    a["ug"][0][op] = np.maximum(jet, 1.5 + 3.0 * w + 0.3 * _modes(rng, shape))[op]
    for q in (1, 2):
        a["ug"][q][op] = (0.8 * _modes(rng, shape))[op]
    a["gf"][3][op] = (200.0 * (1.0 + 0.2 * _modes(rng, shape)))[op]
    a["gf"][4][op] = (1.5e5 * (1.0 + 0.2 * _modes(rng, shape)))[op]
    return f


def _perturbed(case: Case, rng) -> Fields:
    """A restart's fields with seeded smooth changes of up to a few percent."""
    f = case.initial_fields()
    shape = case.ibcell().shape
    op = (case.ibcell() <= 0).astype(np.float64)
    a = f.arrays
    for q in range(3):
        a["ug"][q] *= 1.0 + 0.03 * op * _modes(rng, shape)
    for q in (3, 4):
        a["gf"][q] *= 1.0 + 0.05 * op * _modes(rng, shape)
    a["t"] *= 1.0 + 0.01 * op * _modes(rng, shape)
    return f


def _grid_case(grid: str, seed: int, **kw):
    """(case, start fields) of a furnace or a shipped case."""
    rng = np.random.default_rng(seed)
    if "x" in grid:
        case = _furnace(grid, seed)
        return case, _through_flow(case, rng)
    case, _ = _shipped(grid, wall_sink=True, rad_emission=True, kappa=[0.5] * 10, **kw)
    return case, _perturbed(case, rng)


class Readback:
    """Pinned host buffers for a handle's fields, and the read into them."""

    def __init__(self, solver: GpuSolver, names, single: bool):
        case = solver.case
        shp = (case.lp, case.np, case.mp)
        shapes = {"ug": (3,) + shp, "gf": (9,) + shp, "qa": tuple(s // 2 for s in shp), "qe": tuple(s // 2 for s in shp)}
        self.solver = solver
        self.c = abi.GfmFields()
        self.host = {n: torch.zeros(shapes.get(n, shp), dtype=torch.float64, pin_memory=True) for n in names}
        self.single = {n: torch.zeros(t.shape, dtype=torch.float32) for n, t in self.host.items()} if single else None
        for n, t in self.host.items():
            setattr(self.c, n, abi.dptr(t.numpy()))

    def __call__(self) -> dict:
        self.solver._check(self.solver.lib.gfm_gpu_download(self.solver.h, C.byref(self.c)))
        if self.single is None:
            return dict(self.host)
        for n, t in self.host.items():
            self.single[n].copy_(t)
        return dict(self.single)


def _pinned(f: Fields) -> Fields:
    for k, v in f.arrays.items():
        t = torch.empty(v.shape, dtype=torch.float64, pin_memory=True)
        t.numpy()[...] = v
        f.arrays[k] = t.numpy()
    return f


def _solver(case: Case, c: dict) -> GpuSolver:
    return GpuSolver(case, adi_mode=ADI[c.get("adi", "redblack")], precision=PREC[c["prec"]], bgcon=1.0e-30)


def prepare(c: dict, seed: int) -> State:
    kind = c["kind"]
    rng = np.random.default_rng(seed + 17)
    single = c.get("prec") == "mixed"
    if kind in ("flow", "start"):
        case, f = _grid_case(c["grid"], seed)
        s = _solver(case, c)
        back = Readback(s, STATE, single)
        if kind == "start":
            f = _pinned(f)
            return State(kind=kind, solver=s, back=back, iters=c["iters"], fields=f, c=f.to_c())
        s.upload(f)
        s.initsv()
        return State(kind=kind, solver=s, back=back, iters=c["iters"])
    if kind == "batch":
        solvers, backs = [], []
        for cfg in configs.batch_variants(c["variants"], seed=c["set"]):
            case = Case(dataclasses.replace(cfg, **RUN))
            s = _solver(case, c)
            s.upload(_through_flow(case, rng))
            s.initsv()
            solvers.append(s)
            backs.append(Readback(s, STATE, single))
        return State(kind=kind, solvers=solvers, backs=backs, iters=c["iters"])
    if kind == "radiation":
        if "x" in c["grid"]:
            case, minor = _furnace(c["grid"], seed), None
            f = _through_flow(case, rng)
            f.arrays["t"] *= 1.0 + 0.1 * (case.ibcell() <= 0) * _modes(rng, f.arrays["t"].shape)
        else:
            case, minor = _shipped(c["grid"], minor=True, wall_sink=True, gas_model=True)
            f = _perturbed(case, rng)
        s = _solver(case, c)
        s.upload(f)
        if minor is not None:
            s.initsv()
            s.minor_upload(minor)
        s.wall_setup()
        return State(kind=kind, solver=s, back=Readback(s, ("qa", "qe", "t"), single))
    if kind == "emission":
        case, f, _ = _emission_case(c, seed)
        s = _solver(case, c)
        s.upload(f)
        return State(kind=kind, solver=s, back=Readback(s, ("qe",), single))
    if kind == "msflow":
        case, minor = _shipped(c["grid"], minor=True, wall_sink=True, gas_model=True)
        s = _solver(case, c)
        s.upload(_perturbed(case, rng))
        s.initsv()
        for q in range(minor.gfm.shape[0]):
            minor.gfm[q] *= 1.0 + 0.01 * _modes(rng, minor.gfm[q].shape)
        s.minor_upload(minor)
        s.initsvm(restart=True)
        return State(kind=kind, solver=s, iters=c["iters"])
    if kind == "adlbl3":
        case, sysm, rng6 = _line_system(c, seed)
        return State(kind=kind, solver=_solver(case, c), system=sysm, range=rng6, sweeps=c["sweeps"], single=single)
    # learned
    dims, p, x, target = _learned_inputs(c, seed)
    lp = LearnedPressure(dims, seed=1)
    lp.set_params(p)
    feats = torch.tensor(x, dtype=torch.bfloat16, device="cuda").contiguous()
    return State(kind=kind, lp=lp, feats=feats, target=torch.tensor(target, dtype=torch.float32, device="cuda"), dims=dims)


# ---- one pass ----------------------------------------------------------------

def run(s: State):
    if s.kind == "flow":
        s.solver.gflow(s.iters)
        return s.back()
    if s.kind == "start":
        s.solver._check(s.solver.lib.gfm_gpu_upload(s.solver.h, C.byref(s.c)))
        s.solver.initsv()
        s.solver.gflow(s.iters)
        return s.back()
    if s.kind == "batch":
        gflow_batch(s.solvers, s.iters)
        return [b() for b in s.backs]
    if s.kind == "radiation":
        s.solver.rad_transfer()
        out = s.back()
        for n in ("b_t", "radiosity", "qrs"):
            out[n] = s.solver.wall_array(n)
        return out
    if s.kind == "emission":
        s.solver.rad_emission()
        return s.back()
    if s.kind == "msflow":
        s.solver.msflow(s.iters)
        m = s.solver.minor_download()
        return {"gfm": m.gfm, "smf": m.smf, "rrms": m.rrms}
    if s.kind == "adlbl3":
        xt, ap, as6, bs = s.system
        x = s.solver.adlbl3(xt, ap, as6, bs, *s.range, s.sweeps)
        return x.astype(np.float32) if s.single else x
    loss = s.lp.train_step(s.feats, s.target, s.dims, lr=1.0e-3)
    return {"loss": loss, "params": s.lp.params()}


# ---- what a pass cannot do without ---------------------------------------------

def _sizes(grid: str):
    """(open cells, doubled-grid positions, patches) of a grid."""
    if grid == "0041":
        return 4407, 40 * 48 * 36, 1628
    if grid == "1207":
        return 8263, 172 * 52 * 32, 3500
    nx, ny, nz = (int(v) for v in grid.split("x"))
    return nx * ny * nz, (2 * nx + 4) * (2 * ny + 4) * (2 * nz + 4), 2 * (nx * ny + ny * nz + nx * nz)


def _flow_work(cells, pos, prec, iters):
    # An iteration reads and writes the state (21 fields on the doubled grid)
    # once; its line solves visit a cell 82 times at 24 multiply-adds, and the
    # assembly of 12 equations takes about 2,000 operations a cell.
    w = 4 if prec == "mixed" else 8
    return {"bytes": 2.0 * 21 * pos * w * iters + 14.0 * 8 * pos, "flops": (82 * 48.0 + 2000.0) * cells * iters}


def work(c: dict) -> dict:
    kind = c["kind"]
    if kind == "batch":
        tot = {"bytes": 0.0, "flops": 0.0}
        for _ in range(c["variants"]):   # the variants' mean extents
            w = _flow_work(80 * 40 * 30, 164 * 84 * 64, c["prec"], c["iters"])
            tot = {k: tot[k] + w[k] for k in tot}
        return tot
    cells, pos, nb = _sizes(c["grid"])
    if kind in ("flow", "start"):
        w = _flow_work(cells, pos, c["prec"], c["iters"])
        if kind == "start":
            w["bytes"] += 21.0 * 8 * pos
        return w
    if kind == "radiation":
        # every emitter reaches every cell in each band (10 bands), and one
        # sweep of the exchange reads the view factors (8 bytes) once
        return {"bytes": 3.0 * 8 * pos + 8.0 * nb * nb, "flops": 10.0 * 4 * cells * cells + 2.0 * nb * nb}
    if kind == "emission":
        w = 4 if c["prec"] == "mixed" else 8
        return {"bytes": (w + 8.0) * cells, "flops": 3 * 12 * 15.0 * cells}
    if kind == "msflow":
        return {"bytes": 2.0 * 8 * pos * 9 * c["iters"], "flops": 8 * 400.0 * cells * c["iters"]}
    if kind == "adlbl3":
        return {"bytes": 10.0 * 8 * pos, "flops": 4 * 24 * 2.0 * cells * c["sweeps"] / 2}
    macs = 27.0 * cells * (16 * 16 + 16 * 16 + (16 * 32 + 32 * 32) / 8 + 48 * 16 + 16 * 16)
    return {"bytes": 36.0 * cells + 16.0 * 70512, "flops": 6.0 * macs}


# ---- the same in 64 bits ---------------------------------------------------------

def exact(c: dict, seed: int):
    """Plain 64-bit values: the emission source, the line solve and the
    network's loss and updated parameters.  The whole iteration, the transfer and
    MSFLOW have no short restatement."""
    if c["kind"] == "emission":
        return _exact_emission(c, seed)
    if c["kind"] == "adlbl3":
        return _exact_adlbl3(c, seed)
    if c["kind"] == "learned":
        return _exact_learned(c, seed)
    return None


def _emission_case(c: dict, seed: int):
    rng = np.random.default_rng(seed + 29)
    case = _furnace(c["grid"], seed)
    f = case.initial_fields()
    t = f.arrays["t"]
    t *= 1.0 + 0.25 * _modes(rng, t.shape)
    return case, f, t


def _exact_emission(c: dict, seed: int):
    case, f, t = _emission_case(c, seed)
    g, p = case.grid, case.params
    if c["prec"] == "mixed":
        t = t.astype(np.float32).astype(np.float64)   # what the mixed path is given
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    tk = torch.tensor(t[1::2, 1::2, 1::2] * p.t0, device=dev)
    op = torch.tensor(case.ibcell()[1::2, 1::2, 1::2] <= 0, device=dev) & (tk >= 300.0)
    ax = lambda ptr, n: torch.tensor(np.ctypeslib.as_array(ptr, shape=(n,))[1::2].copy(), device=dev)
    dx, dr, dz = ax(g.dx, case.mp)[None, None, :], ax(g.dr, case.np)[None, :, None], ax(g.dz, case.lp)[:, None, None]
    vol = dx * dr * ax(g.rs, case.np)[None, :, None] * dz
    sa = 2.0 * (dx * dr + dr * dz + dx * dz)
    opl = 6.0 * vol / sa
    tsafe = torch.where(op, tk, torch.full_like(tk, 1000.0))
    s = torch.zeros_like(tk)
    low = torch.zeros_like(tk)
    for l in range(g.nwl):
        if l < g.nwl - 1:
            x = (p.hck / p.ri / g.wl[l]) / tsafe
            frac = torch.zeros_like(tk)
            for n in range(1, 400):   # fraction of the black-body emission below the band edge
                term = (x ** 3 / n + 3 * x ** 2 / n ** 2 + 6 * x / n ** 3 + 6.0 / n ** 4) * torch.exp(-n * x)
                frac += term
                if float(term.max()) < 1.0e-18:
                    break
            frac = (frac * 15.0 / math.pi ** 4).clamp(max=1.0)
            deb = frac - low
            thin = deb <= 1.0e-3
            deb = torch.where(thin, torch.zeros_like(deb), deb)
            low = torch.where(thin, low, frac)
        else:
            deb = 1.0 - low
        x0 = g.akl0[l] * opl
        x1 = 1.0e-3
        s = s + deb * torch.where(x0 <= x1, x0 * ((1.0 - math.exp(-x1)) / x1), -torch.expm1(-x0))
    qe = torch.where(op, sa * p.sig * p.ri ** 2 * tk ** 4 * s, torch.zeros_like(tk))
    return {"qe": qe.cpu()}


def _line_system(c: dict, seed: int):
    """A diagonally dominant system on the cell centres, as the solver's own
    equations are, with a smooth right-hand side; start and border seeded."""
    rng = np.random.default_rng(seed)
    case = _furnace(c["grid"], seed)
    shp = (case.lp, case.np, case.mp)
    inner = (slice(3, case.lp - 2, 2), slice(3, case.np - 2, 2), slice(3, case.mp - 2, 2))
    n = tuple(len(range(*sl.indices(m))) for sl, m in zip(inner, shp))
    ap, bs, xt, as6 = np.ones(shp), np.zeros(shp), np.zeros(shp), [np.zeros(shp) for _ in range(6)]
    a = rng.uniform(0.1, 1.0, (6,) + n)
    for q in range(6):
        as6[q][inner] = a[q]
    ap[inner] = a.sum(axis=0) * 1.05
    bs[inner] = _modes(rng, n) + 0.1 * rng.standard_normal(n)
    whole = (slice(1, case.lp, 2), slice(1, case.np, 2), slice(1, case.mp, 2))
    xt[whole] = 0.1 * rng.standard_normal(xt[whole].shape)
    return case, (xt, ap, as6, bs), (4, case.mp - 2, 4, case.np - 2, 4, case.lp - 2)


def _thomas(ap, sub, nxt, rhs, lo, hi, free):
    """Lines along the last axis: x_r AP = AS_sub x_(r-1) + AS_next x_(r+1) + rhs; rows not `free` keep rhs."""
    pt, qt = torch.zeros_like(ap), torch.zeros_like(ap)
    pp, qq = torch.zeros_like(lo), lo
    for r in range(ap.shape[-1]):
        d = ap[..., r] - pp * sub[..., r]
        pp = torch.where(free[..., r], nxt[..., r] / d, torch.zeros_like(d))
        qq = torch.where(free[..., r], (rhs[..., r] + sub[..., r] * qq) / d, rhs[..., r])
        pt[..., r], qt[..., r] = pp, qq
    x, v = torch.empty_like(qt), hi
    for r in range(ap.shape[-1] - 1, -1, -1):
        v = qt[..., r] + pt[..., r] * v
        x[..., r] = v
    return x


def _exact_adlbl3(c: dict, seed: int):
    case, (xt, ap, as6, bs), rg = _line_system(c, seed)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    whole = (slice(1, case.lp, 2), slice(1, case.np, 2), slice(1, case.mp, 2))
    if c["prec"] == "mixed":   # what the mixed path is given
        xt, ap, bs, as6 = (v.astype(np.float32).astype(np.float64) for v in (xt, ap, bs, np.stack(as6)))
    t = lambda v: torch.tensor(np.ascontiguousarray(np.transpose(v[whole], (2, 1, 0))), device=dev)   # (I, J, K)
    x, ap, bs, a = t(xt), t(ap), t(bs), [t(v) for v in as6]
    free = torch.tensor(np.ascontiguousarray(np.transpose(case.ibcell()[whole] < 1, (2, 1, 0))), device=dev)
    i = slice(1, -1)
    ap, bs, a, free = ap[i, i, i], bs[i, i, i], [v[i, i, i] for v in a], free[i, i, i]
    T = lambda v: v.transpose(-1, -2).contiguous()
    for _ in range(2 * c["sweeps"]):
        for colour in (0, 1):
            k = slice(colour, None, 2)
            A = [v[k] for v in a]
            P, F = ap[k], free[k]
            bx = bs[k] + A[1] * x[2:, i, i][k] + A[0] * x[:-2, i, i][k]
            for _pass in range(2):
                b = x[1:-1][k]   # the planes of the colour, with their border
                old = b[:, i, i]
                ry = torch.where(F, bx + A[5] * b[:, i, 2:] + A[4] * b[:, i, :-2], old)
                rz = torch.where(F, bx + A[3] * b[:, 2:, i] + A[2] * b[:, :-2, i], old)
                xy = T(_thomas(T(P), T(A[2]), T(A[3]), T(ry), b[:, 0, i], b[:, -1, i], T(F)))
                xz = _thomas(P, A[4], A[5], rz, b[:, i, 0], b[:, i, -1], F)
                n = x.clone()
                n[1:-1][k, 1:-1, 1:-1] = 0.5 * (xy + xz)
                x = n
    out = xt.copy()
    out[whole] = np.transpose(x.cpu().numpy(), (2, 1, 0))
    return out


_LAYERS = ((16, 16), (16, 16), (16, 32), (32, 32), (48, 16), (16, 16))


def _learned_inputs(c: dict, seed: int):
    """Parameters, features (scaled right-hand side, open mask) and target."""
    rng = np.random.default_rng(seed)
    nx, ny, nz = dims = tuple(int(v) for v in c["grid"].split("x"))
    parts = []
    for l, (ci, co) in enumerate(_LAYERS):
        a = math.sqrt(6.0 / (27 * ci))
        w = rng.uniform(-a, a, (27, co, ci))
        b = rng.uniform(-0.05, 0.05, co)
        if l == 0:
            w[:, :, 2:] = 0.0       # two input channels are in use
        if l == 5:
            w[:, 1:, :] = 0.0       # one output channel is
            b[1:] = 0.0
        parts += [w.reshape(-1), b]
    p = np.concatenate(parts).astype(np.float32)
    x = np.zeros((nz, ny, nx, 16), np.float32)
    x[..., 1] = 1.0
    x[: max(1, nz // 8), : max(1, ny // 6), : max(1, nx // 8), 1] = 0.0   # a blocked corner
    rhs = _modes(rng, (nz, ny, nx), n=6, kmax=6) + 0.3 * rng.standard_normal((nz, ny, nx))
    x[..., 0] = np.where(x[..., 1] > 0, rhs / rhs.std(), 0.0)
    target = _modes(rng, (nz, ny, nx), n=6)
    target = np.where(x[..., 1] > 0, target / target.std(), 0.0)
    return dims, p, x.reshape(-1, 16), target.reshape(-1).astype(np.float32)


def _exact_learned(c: dict, seed: int):
    dims, p, x, target = _learned_inputs(c, seed)
    nx, ny, nz = dims
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    x = torch.tensor(x).to(torch.bfloat16).double().to(dev).reshape(nz, ny, nx, 16).permute(3, 0, 1, 2)[None]
    target = torch.tensor(target, dtype=torch.float64, device=dev).reshape(nz, ny, nx)
    w, off = [], 0
    flat = torch.tensor(p, dtype=torch.float64, device=dev, requires_grad=True)
    for ci, co in _LAYERS:
        k = flat[off: off + 27 * ci * co].reshape(3, 3, 3, co, ci).permute(3, 4, 0, 1, 2)
        off += 27 * ci * co
        w.append((k, flat[off: off + co]))
        off += co

    def conv(v, l):
        # 27 shifted products: a convolution in 64 bits on any device
        k, b = w[l]
        v = torch.nn.functional.pad(v, (1,) * 6)
        out = b[None, :, None, None, None]
        d, h, m = v.shape[2] - 2, v.shape[3] - 2, v.shape[4] - 2
        for z in range(3):
            for y in range(3):
                for q in range(3):
                    out = out + torch.einsum("oc,ncdhw->nodhw", k[:, :, z, y, q], v[:, :, z: z + d, y: y + h, q: q + m])
        return out
    relu = torch.relu
    e0 = relu(conv(relu(conv(x, 0)), 1))
    e1 = relu(conv(relu(conv(torch.nn.functional.avg_pool3d(e0, 2), 2)), 3))
    up = e1.repeat_interleave(2, 2).repeat_interleave(2, 3).repeat_interleave(2, 4)
    out = conv(relu(conv(torch.cat([e0, up], 1), 4)), 5)[0, 0]
    op = x[0, 1] > 0.5
    loss = torch.where(op, (out - target) ** 2, torch.zeros_like(out)).sum() / op.sum()
    loss.backward()
    # Adam's first step from zero moments (0.9, 0.999, 1e-8) at the pass's rate
    g = flat.grad
    params = flat.detach() - 1.0e-3 * g / (g.abs() + 1.0e-8)
    return {"loss": float(loss), "params": params.cpu().numpy()}
