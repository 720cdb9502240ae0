"""The plane visits of the line solver (adi_visit.cu) at the edges of their
forms: the smallest and odd planes, planes on both sides of each form's size,
planes beyond every form (the segmented passes, the line-by-line march), and
lines whose elimination from both ends meets a vanishing pivot.  Two sweeps on
manufactured systems against the oracle in the same plane order; tolerances of
test_gpu_adi (1e-13 FP64, 1e-5 mixed)."""
import numpy as np
import pytest

from gfm_gb300 import Case, GpuSolver, abi, configs
from gfm_gb300.solver import GfmError

from .test_gpu_adi import _oracle_adlbl3
from .test_oracle_adi import manufactured

pytestmark = pytest.mark.gpu

TOL = {abi.GFM_PREC_FP64: 1e-13, abi.GFM_PREC_MIXED: 1e-5}


def _compare(case, adi, prec, system, rng, open_):
    ap, as6, bs, x0 = system
    g = GpuSolver(case, adi_mode=adi, precision=prec)
    xg = g.adlbl3(x0, ap, as6, bs, *rng, 2)
    g.close()
    xo = _oracle_adlbl3(case, adi, ap, as6, bs, x0, rng, 2)
    err = np.abs(xg - xo)[open_].max() / np.abs(xo[open_]).max()
    assert err < TOL[prec], err


# points a plane: 16 .. 512 | 1024 | 2048 | 4096 | 6144 | larger (FP32 forms;
# FP64 has 512 | 1024 | larger), and planes beyond shared memory in FP64
@pytest.mark.parametrize("prec", [abi.GFM_PREC_FP64, abi.GFM_PREC_MIXED])
@pytest.mark.parametrize("adi", [abi.GFM_ADI_REDBLACK, abi.GFM_ADI_MARCH])
@pytest.mark.parametrize("ny,nz", [(4, 4), (5, 9), (33, 15), (16, 32), (27, 19), (32, 32), (41, 31), (64, 32), (69, 30),
                                   (64, 64), (65, 64), (96, 64), (97, 65), (150, 96)])
def test_plane_sizes_match_the_oracle(ny, nz, adi, prec):
    case = Case(configs.tiny_furnace(5, ny, nz))
    ap, as6, bs, x0, sol, rng, open_ = manufactured(case)
    _compare(case, adi, prec, (ap, as6, bs, x0), rng, open_)


# FP32 visits by where their records are staged: both directions' in shared
# memory with segments of at most 4 rows (25x30 and, on 768 threads, 72x10) and
# of more (40x24 with more planes than SMs, 50x28), one direction's at a time
# (96x60, 63x64, 31x190), one direction's but for a last row (192x32)
@pytest.mark.parametrize("nx,ny,nz", [(7, 25, 30), (400, 40, 24), (7, 72, 10), (9, 50, 28), (90, 96, 60), (9, 63, 64),
                                      (5, 192, 32), (6, 31, 190)])
def test_fp32_visits_match_the_oracle_where_their_records_are_staged(nx, ny, nz):
    case = Case(configs.tiny_furnace(nx, ny, nz))
    ap, as6, bs, x0, sol, rng, open_ = manufactured(case)
    _compare(case, abi.GFM_ADI_REDBLACK, abi.GFM_PREC_MIXED, (ap, as6, bs, x0), rng, open_)


# two open cells coupled only to each other along y (or z): the second one met
# by an elimination has a zero pivot, which the reference copies; at the two
# ends of the lines and across their middle
@pytest.mark.parametrize("prec", [abi.GFM_PREC_FP64, abi.GFM_PREC_MIXED])
@pytest.mark.parametrize("adi", [abi.GFM_ADI_REDBLACK, abi.GFM_ADI_MARCH])
@pytest.mark.parametrize("along", ["y", "z"])
def test_vanishing_pivots_are_the_references(along, adi, prec):
    case = Case(configs.tiny_furnace(6, 12, 10))
    ap, as6, bs, x0, sol, rng, open_ = manufactured(case)
    ib0, ie, jb, je, kb, ke = rng
    i = ib0 + 2
    ax, lo, hi = (1, jb, je) if along == "y" else (2, kb, ke)
    n = (hi - lo) // 2 + 1
    for q, r in enumerate((0, n // 2 - 1, n // 2, n - 2)):   # the pair (r, r+1) of line q
        for step, (sub, nxt) in ((0, (0.0, 0.5)), (1, (0.5, 0.0))):
            pos = [i, jb + 4 + 2 * q, kb + 4 + 2 * q]
            pos[ax] = lo + 2 * (r + step)
            at = (pos[2] - 1, pos[1] - 1, pos[0] - 1)
            if case.ibcell()[at] > 0:
                continue
            for a in as6:
                a[at] = 0.0
            as6[2 * ax][at], as6[2 * ax + 1][at] = sub, nxt
            ap[at], bs[at] = 0.5, 0.01 * (2 * step - 1)
    _compare(case, adi, prec, (ap, as6, bs, x0), rng, open_)


# four rows coupled only to each other along y (or z), well conditioned (73) but not
# dominated by their diagonal: the lower two are singular up to rounding, so an
# elimination from the line's far end loses the result (errors of the size of the
# solution), and only the reference's order keeps it.  Across the lines' middle, at
# their end and at their start, with both signs of the third row's coupling.  The
# oracle's rounding and the kernel's, 73 units each through four passes.
@pytest.mark.parametrize("prec,unit", [(abi.GFM_PREC_FP64, 2.0 ** -53), (abi.GFM_PREC_MIXED, 2.0 ** -24)])
@pytest.mark.parametrize("adi", [abi.GFM_ADI_REDBLACK, abi.GFM_ADI_MARCH])
@pytest.mark.parametrize("along", ["y", "z"])
def test_lines_without_dominance_keep_the_references_order(along, adi, prec, unit):
    case = Case(configs.tiny_furnace(6, 12, 11))
    ap, as6, bs, x0, sol, rng, open_ = manufactured(case)
    ax, lo, hi = (1, rng[2], rng[3]) if along == "y" else (2, rng[4], rng[5])
    n = (hi - lo) // 2 + 1
    placed = 0
    for i in (rng[0] + 2, rng[0] + 4):
        for q, r in enumerate((n - n // 2 - 2, n - 4, 0)):   # rows r .. r+3 of line q
            for sign in (-1.0, 1.0):
                pos = [i, rng[2] + 2 * (2 * q + (sign > 0)), rng[4] + 2 * (2 * q + (sign > 0))]
                at = []
                for step in range(4):
                    pos[ax] = lo + 2 * (r + step)
                    at.append((pos[2] - 1, pos[1] - 1, pos[0] - 1))
                if any(case.ibcell()[a] > 0 for a in at):
                    continue
                placed += 1
                rows = ((4.0, 0.0, 1.0), (4.0, 1.0, 1.0), (0.3, sign, 0.1), (0.3, 0.9, 0.0))
                for step, (p, sub, nxt) in enumerate(rows):
                    for a in as6:
                        a[at[step]] = 0.0
                    as6[2 * ax][at[step]], as6[2 * ax + 1][at[step]] = sub, nxt
                    ap[at[step]], bs[at[step]] = p, 1.0 + step
    assert placed >= 8
    g = GpuSolver(case, adi_mode=adi, precision=prec)
    xg = g.adlbl3(x0, ap, as6, bs, *rng, 1)
    g.close()
    xo = _oracle_adlbl3(case, adi, ap, as6, bs, x0, rng, 1)
    err = np.abs(xg - xo)[open_].max() / np.abs(xo[open_]).max()
    assert err < 4 * 2 * 73 * unit, err


# visits read a call's records before the visit ahead of them has ended: calls with
# other coefficients one after the other on one handle give the bits of a handle of
# their own without programmatic launch
@pytest.mark.parametrize("prec", [abi.GFM_PREC_FP64, abi.GFM_PREC_MIXED])
def test_records_of_the_call_before_are_not_met(prec, monkeypatch):
    case = Case(configs.tiny_furnace(30, 24, 20))
    systems = [manufactured(case, seed=s) for s in (7, 8, 9)]

    def solve(g, s):
        ap, as6, bs, x0, sol, rng, open_ = s
        return g.adlbl3(x0, ap, as6, bs, *rng, 3)

    g = GpuSolver(case, adi_mode=abi.GFM_ADI_REDBLACK, precision=prec)
    got = [solve(g, s) for s in systems * 3]
    g.close()
    monkeypatch.setenv("GFM_PDL", "0")
    for k, s in enumerate(systems):
        g = GpuSolver(case, adi_mode=abi.GFM_ADI_REDBLACK, precision=prec)
        want = solve(g, s)
        g.close()
        assert all(np.array_equal(x, want) for x in got[k::3])


# a visit whose wait for its plane, or for its records, runs out (here at once: no
# poll of the barrier) is reported, by a line solve and by an iteration, and the GPU
# goes on; records of both directions staged (25x30), of one at a time (96x60)
@pytest.mark.parametrize("polls", ["0,1000000", "1000000,0"])
@pytest.mark.parametrize("ny,nz", [(25, 30), (96, 60)])
def test_a_wait_that_runs_out_is_reported(ny, nz, polls, monkeypatch):
    case = Case(configs.tiny_furnace(9, ny, nz))
    ap, as6, bs, x0, sol, rng, open_ = manufactured(case)
    solve = lambda g: g.adlbl3(x0, ap, as6, bs, *rng, 2)
    kw = dict(adi_mode=abi.GFM_ADI_REDBLACK, precision=abi.GFM_PREC_MIXED)
    g = GpuSolver(case, **kw)
    want = solve(g)
    monkeypatch.setenv("GFM_ADI_POLLS", polls)
    monkeypatch.setenv("GFM_RB_TUNE", "0")   # the plane visits
    h = GpuSolver(case, **kw)
    with pytest.raises(GfmError, match="did not arrive") as e:
        solve(h)
    assert e.value.rc == abi.GFM_E_TIMEOUT
    h.start()
    with pytest.raises(GfmError, match="did not arrive"):
        h.gflow(1)
    h.close()
    assert np.array_equal(solve(g), want)
    g.close()


# the march's two forms share a memory: four field-sized arrays a system, as the
# line-by-line form alone needs (red-black: 23 class-sized ones)
def test_march_scratch_is_one_forms():
    import torch
    case = Case(configs.tiny_furnace(96, 48, 32))
    hx, hy, hz = case.mp // 2 + 1, case.np // 2 + 1, case.lp // 2 + 1
    up = lambda n: (n + 15) // 16 * 16
    ns, nh = 8 * up(hx) * hy * hz, 2 * up((hx + 1) // 2) * hy * hz

    def used(adi):
        free = torch.cuda.mem_get_info()[0]
        g = GpuSolver(case, adi_mode=adi)
        u = free - torch.cuda.mem_get_info()[0]
        g.close()
        return u

    used(abi.GFM_ADI_REDBLACK)   # the context and the module
    more = used(abi.GFM_ADI_MARCH) - used(abi.GFM_ADI_REDBLACK)
    assert more <= 8 * 8 * (max(4 * ns, 19 * nh) - 23 * nh) + (64 << 20), more


_MARCH_FORMS = """
import hashlib, sys
sys.path.insert(0, {root!r})
import numpy as np
from gfm_gb300 import Case, GpuSolver, abi, configs
from tests.test_oracle_adi import manufactured
h = hashlib.sha256()
for ny, nz in ((12, 9), (33, 31), (41, 50)):
    case = Case(configs.tiny_furnace(6, ny, nz))
    ap, as6, bs, x0, sol, rng, open_ = manufactured(case)
    ap[:, : case.np // 2] *= 0.4   # half of the lines without a dominant diagonal
    for prec in (abi.GFM_PREC_FP64, abi.GFM_PREC_MIXED):
        g = GpuSolver(case, adi_mode=abi.GFM_ADI_MARCH, precision=prec)
        x = g.adlbl3(x0, ap, as6, bs, *rng, 2)
        g.close()
        assert np.isfinite(x).all()
        h.update(x.tobytes())
print(h.hexdigest())
"""


# the march's three forms -- plane visit, and line by line with 4 rows a batch or 1 --
# give the same bits, in either order of elimination (a process each: the variable is
# read once)
def test_march_forms_give_the_same_bits():
    import os
    import pathlib
    import subprocess
    import sys
    code = _MARCH_FORMS.format(root=str(pathlib.Path(__file__).resolve().parents[1]))
    out = []
    for rows in (None, "4", "1"):
        env = {k: v for k, v in os.environ.items() if k != "GFM_MARCH_ROWS"} | ({"GFM_MARCH_ROWS": rows} if rows else {})
        r = subprocess.run([sys.executable, "-c", code], env=env, capture_output=True, text=True, timeout=600)
        assert r.returncode == 0, r.stderr
        out.append(r.stdout.strip().splitlines()[-1])
    assert out[0] == out[1] == out[2]


def _adlbl3(ap, as6, bs, x0, nim, dt):
    """ADLBL3 in the reference's plane order with the reference's expressions in dtype `dt`, arrays (plane, J, K)
    with a border of one point."""
    a, ap, bs, x = [q.astype(dt) for q in as6], ap.astype(dt), bs.astype(dt), x0.astype(dt)
    c = slice(1, -1)

    def lines(p, rhs, sub, nxt, v):   # rows along the first axis
        pt, q = np.zeros((v.shape[0], v.shape[1] - 2), dt), np.zeros((v.shape[0], v.shape[1] - 2), dt)
        q[0], out = v[0, c], v[:, c].copy()
        for r in range(1, v.shape[0] - 1):
            alp = p[r] - pt[r - 1] * sub[r]
            pt[r], q[r] = nxt[r] / alp, (rhs[r] + sub[r] * q[r - 1]) / alp
        for r in range(v.shape[0] - 2, 0, -1):
            out[r] = out[r + 1] * pt[r] + q[r]
        return out[1:-1]

    def visit(i):
        for _ in range(2):
            v = x[i]
            b = bs[i] + a[1][i] * x[i + 1] + a[0][i] * x[i - 1]
            ry, rz = b.copy(), b.copy()
            ry[c, c] = b[c, c] + a[5][i][c, c] * v[c, 2:] + a[4][i][c, c] * v[c, :-2]
            rz[c, c] = b[c, c] + a[3][i][c, c] * v[2:, c] + a[2][i][c, c] * v[:-2, c]
            y = lines(ap[i][:, c], ry[:, c], a[2][i][:, c], a[3][i][:, c], v)
            z = lines(ap[i].T[:, c], rz.T[:, c], a[4][i].T[:, c], a[5][i].T[:, c], v.T).T
            x[i][c, c] = (y + z) / dt(2)

    n = x.shape[0] - 2
    for _ in range(nim):
        for i in [*range(1, n + 1), *range(n, 0, -1)]:
            visit(i)
    return x


# The rounding error of the march's solution against extended precision, root mean
# square over four systems: at most that of the reference's expressions in the same
# precision (an exact emulation of the roundings gives 0.96 to 0.98 of it; with AL, PT
# and the right-hand sides as products by 1/ALP 1.05).
@pytest.mark.parametrize("prec", [abi.GFM_PREC_FP64, abi.GFM_PREC_MIXED])
def test_rounding_errors_of_the_march_are_at_most_the_references(prec):
    case = Case(configs.tiny_furnace(20, 24, 20))
    shp = (case.lp, case.np, case.mp)
    dt = np.float64 if prec == abi.GFM_PREC_FP64 else np.float32
    inner = (slice(3, case.lp - 2, 2), slice(3, case.np - 2, 2), slice(3, case.mp - 2, 2))
    outer = (slice(1, case.lp, 2), slice(1, case.np, 2), slice(1, case.mp, 2))
    assert (case.ibcell()[inner] <= 0).all()
    se = sr = 0.0
    g = GpuSolver(case, adi_mode=abi.GFM_ADI_MARCH, precision=prec)
    for seed in range(4):
        rng = np.random.default_rng(seed)
        n = tuple(len(range(*s.indices(m))) for s, m in zip(inner, shp))
        f32 = lambda v: v.astype(np.float32).astype(np.float64)
        ap, bs, x0, as6 = np.ones(shp), np.zeros(shp), np.zeros(shp), [np.zeros(shp) for _ in range(6)]
        a = f32(rng.uniform(0.1, 1.0, (6,) + n))
        for q in range(6):
            as6[q][inner] = a[q]
        ap[inner], bs[inner] = f32(1.05 * a.sum(axis=0)), f32(rng.standard_normal(n))
        x0[outer] = f32(rng.standard_normal(x0[outer].shape))
        x = g.adlbl3(x0, ap, as6, bs, 4, case.mp - 2, 4, case.np - 2, 4, case.lp - 2, 2)[outer].transpose(2, 1, 0)
        cut = lambda v: v[outer].transpose(2, 1, 0)
        args = (cut(ap), [cut(q) for q in as6], cut(bs), cut(x0), 2)
        exact = _adlbl3(*args, np.longdouble)
        se += float(((x - exact) ** 2).sum())
        sr += float(((_adlbl3(*args, dt) - exact) ** 2).sum())
    g.close()
    assert se <= sr, (se / sr) ** 0.5
