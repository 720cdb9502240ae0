"""Volume radiation transfer on the GPU against the CPU oracle, through the C
ABI (gfm_gpu_rad_transfer vs gfo_rad_transfer) on the same uploaded state.

Per emitter the kernel follows the oracle's operation order, with the same
angle function, so the branch decisions agree; QAL is summed per CTA and then
over the CTAs, so QA differs from the oracle's single running sum by the
association of the additions only.  Tolerances: QE 1e-13 relative per cell
(band fractions and EMF use the device's exp), QA 1e-11 relative per cell
above 1e-9 of the largest value, totals 1e-11 relative."""
import numpy as np
import pytest
import torch

from gfm_gb300 import Case, GpuSolver, abi, configs
from oracle.pyoracle import Oracle

pytestmark = pytest.mark.gpu


def _state(cfg, iters):
    case = Case(cfg)
    o = Oracle(case)
    o.initsv()
    o.gflow(iters)
    return case, o


def _compare(fg, fo, tg, to):
    qe_g, qe_o = fg.arrays["qe"], fo.arrays["qe"]
    qa_g, qa_o = fg.arrays["qa"], fo.arrays["qa"]
    assert np.count_nonzero(qe_o) > 0
    big = qe_o > 0
    assert np.all((qe_g > 0) == big)
    assert np.max(np.abs(qe_g[big] - qe_o[big]) / qe_o[big]) < 1e-13
    sel = qa_o > 1e-9 * qa_o.max()
    assert np.all(qa_g[~sel] <= 2e-9 * qa_o.max())
    assert np.max(np.abs(qa_g[sel] - qa_o[sel]) / qa_o[sel]) < 1e-11
    assert tg["n_emitters"] == to["n_emitters"]
    for k in ("qe_sum_from_open", "qa_sum_to_open", "qa_sum_to_wall", "qa_sum_to_inlet", "qa_sum_to_exit",
              "tot_qe_h2o_co2"):
        assert tg[k] == pytest.approx(to[k], rel=1e-11, abs=1e-6), k


@pytest.mark.parametrize("cfg,iters", [
    (configs.tiny_furnace(), 20),
    (configs.tiny_furnace(nx=16, ny=10, nz=8), 12),
    (configs.furnace_variant(3, nx=20, ny=12, nz=10), 8),
])
def test_transfer_matches_oracle(cfg, iters):
    case, o = _state(cfg, iters)
    g = GpuSolver(case, precision=abi.GFM_PREC_FP64)
    g.upload(o.download())
    tg = g.rad_transfer()
    to = o.rad_transfer()
    _compare(g.download(), o.download(), tg, to)
    g.close()
    o.close()


def test_transfer_is_deterministic_and_conserves_energy():
    case, o = _state(configs.tiny_furnace(nx=16, ny=10, nz=8), 12)
    st = o.download()
    out = []
    for _ in range(2):
        g = GpuSolver(case, precision=abi.GFM_PREC_FP64)
        g.upload(st)
        t = g.rad_transfer()
        f = g.download()
        out.append((t, f.arrays["qa"].copy(), f.arrays["qe"].copy()))
        g.close()
    assert out[0][0] == out[1][0]
    assert np.array_equal(out[0][1], out[1][1]) and np.array_equal(out[0][2], out[1][2])
    t = out[0][0]
    absorbed = sum(t[k] for k in ("qa_sum_to_open", "qa_sum_to_wall", "qa_sum_to_inlet", "qa_sum_to_exit",
                                  "qa_sum_to_melt"))
    assert abs(t["qe_sum_from_open"] - absorbed) <= 1e-12 * t["qe_sum_from_open"]
    o.close()


def test_iterations_after_the_transfer_match_the_oracle():
    """The enthalpy source then carries QA - QE (Source.f90:437-439)."""
    case, o = _state(configs.tiny_furnace(), 20)
    g = GpuSolver(case, adi_mode=abi.GFM_ADI_MARCH, precision=abi.GFM_PREC_FP64)
    g.upload(o.download())
    g.rad_transfer()
    o.rad_transfer()
    sg, _ = g.gflow(5)
    so, _ = o.gflow(5)
    fg, fo = g.download(), o.download()
    mask = case.ibcell() <= 0
    for n in ("t", "p"):
        a, b = fg.arrays[n][mask], fo.arrays[n][mask]
        assert np.linalg.norm(a - b) / np.linalg.norm(b) < 1e-9, n
    assert sg["res_mass"] == pytest.approx(so["res_mass"], rel=1e-8)
    g.close()
    o.close()


def test_mixed_precision_transfer_runs_and_conserves_energy():
    case, o = _state(configs.tiny_furnace(nx=16, ny=10, nz=8), 12)
    g = GpuSolver(case, adi_mode=abi.GFM_ADI_REDBLACK, precision=abi.GFM_PREC_MIXED)
    g.upload(o.download())
    t = g.rad_transfer()
    to = o.rad_transfer()
    assert t["n_emitters"] == to["n_emitters"]
    assert t["qe_sum_from_open"] == pytest.approx(to["qe_sum_from_open"], rel=1e-5)
    st, _ = g.gflow(3)
    assert np.isfinite(st["res_mass"])
    g.close()
    o.close()


@pytest.mark.parametrize("kappa,wl_um", [
    (tuple(float(k) for k in np.geomspace(0.05, 5.0, 10)), (1.0, 1.5, 2.0, 3.0, 4.0, 6.0, 8.0, 12.0, 20.0, 1000.0)),
    ((0.3, 1.5), (4.0, 1000.0)),
])
def test_transfer_matches_oracle_for_other_band_sets(kappa, wl_um):
    """10 bands (the count of the 384x160x96 configuration, kappa log-uniform
    on 0.05-5 1/m) and 2 bands take the kernel's other instantiations."""
    cfg = configs.tiny_furnace(nx=16, ny=10, nz=8, kappa=kappa, wl_um=wl_um)
    case, o = _state(cfg, 8)
    g = GpuSolver(case, precision=abi.GFM_PREC_FP64)
    g.upload(o.download())
    tg = g.rad_transfer()
    to = o.rad_transfer()
    _compare(g.download(), o.download(), tg, to)
    g.close()
    o.close()


def test_transfer_with_the_slab_arrays_in_global_memory(monkeypatch):
    """Grids whose slab arrays exceed shared memory (at 192x96x64 the z-slab
    needs 442 KB) keep them in global scratch; forced here on a small grid,
    the same results as the oracle."""
    monkeypatch.setenv("GFM_RAD_GLOBAL_SLAB", "1")
    case, o = _state(configs.tiny_furnace(nx=16, ny=10, nz=8), 12)
    g = GpuSolver(case, precision=abi.GFM_PREC_FP64)
    g.upload(o.download())
    tg = g.rad_transfer()
    to = o.rad_transfer()
    _compare(g.download(), o.download(), tg, to)
    g.close()
    o.close()


def _stretch(case, growth):
    """Cells of the case's box that grow by `growth` along each axis (the box's size kept)."""
    g = case.grid
    for x, dx, n, f in ((g.x, g.dx, g.mp, growth[0]), (g.r, g.dr, g.np, growth[1]), (g.z, g.dz, g.lp, growth[2])):
        size, i = x[n - 1] - x[0], np.arange(n)
        pos = i / (n - 1) if f == 1.0 else (f ** (i / 2) - 1) / (f ** ((n - 1) / 2) - 1)
        x0 = x[0]
        for m in range(n):
            x[m] = x0 + size * pos[m]
        for m in range(1, n - 1):
            dx[m] = x[m + 1] - x[m - 1]


# The angle tables' walks (longer than the first guess of four cells where the
# cells grow away from the emitter), the two block sizes, band counts that do
# and do not divide a warp's lanes, and the ways a CTA's arrays and the tables
# are kept (0: shared memory and all emitters' tables; 2: global scratch and
# tables filled part by part).  Same tolerances as above.
@pytest.mark.parametrize("scratch", ["0", "2"])
@pytest.mark.parametrize("growth", [(1.0, 1.0, 1.0), (1.7, 1.0, 1.15), (0.8, 1.5, 0.6)])
@pytest.mark.parametrize("dims,bands", [((12, 8, 6), 1), ((13, 14, 7), 3), ((12, 37, 6), 16), ((16, 8, 41), 10)])
def test_transfer_over_grids_band_counts_and_scratch(dims, bands, growth, scratch, monkeypatch):
    monkeypatch.setenv("GFM_RAD_GLOBAL_SLAB", scratch)
    kappa = tuple(float(k) for k in np.geomspace(0.05, 5.0, bands)) if bands > 1 else (0.4,)
    wl = tuple(float(w) for w in np.geomspace(1.0, 20.0, bands - 1)) + (1000.0,)
    cfg = configs.tiny_furnace(nx=dims[0], ny=dims[1], nz=dims[2], kappa=kappa, wl_um=wl)
    case, o = _state(cfg, 2)
    st = o.download()
    o.close()
    _stretch(case, growth)
    o = Oracle(case, st)
    g = GpuSolver(case, precision=abi.GFM_PREC_FP64)
    g.upload(st)
    tg = g.rad_transfer()
    to = o.rad_transfer()
    _compare(g.download(), o.download(), tg, to)
    g.close()
    o.close()


def _table_bytes(case, codes=4):
    """Of the angle tables of all directions with walks of at least `codes` codes."""
    n = (case.mp // 2, case.np // 2, case.lp // 2)
    rec = lambda m: (m + 1) * codes + (m + 7) // 8
    return sum(8 * n[d] ** 2 * (n[u] * rec(n[u]) + n[v] * rec(n[v])) for d, u, v in ((0, 1, 2), (1, 0, 2), (2, 0, 1)))


# Where memory is short (a handle's limit in MB) a transfer takes its tables in
# parts; also where the walks are longer than the first guess (stretched cells), of
# which one set is held.
@pytest.mark.parametrize("growth", [(1.0, 1.0, 1.0), (1.7, 1.0, 1.15)])
def test_transfer_takes_its_tables_in_parts_where_memory_is_short(growth, monkeypatch):
    case, o = _state(configs.tiny_furnace(nx=40, ny=30, nz=24), 1)
    st = o.download()
    o.close()
    _stretch(case, growth)

    def transfer(mb):
        monkeypatch.setenv("GFM_DEVICE_MB", str(mb))
        free = torch.cuda.mem_get_info()[0]
        g = GpuSolver(case, precision=abi.GFM_PREC_FP64)
        try:
            g.upload(st)
            t = g.rad_transfer()
            return t, g.download().arrays["qa"], (free - torch.cuda.mem_get_info()[0]) >> 20
        finally:
            g.close()

    tables = _table_bytes(case) >> 20
    assert tables > 100
    transfer(0)   # the context and the module
    whole, qa, used = transfer(0)
    limit = used - int(0.8 * tables)
    parts, qp, short = transfer(limit)
    assert short <= limit + 32
    assert parts["n_emitters"] == whole["n_emitters"]
    assert parts["qa_sum_to_open"] == pytest.approx(whole["qa_sum_to_open"], rel=1e-11)
    sel = qa > 1e-9 * qa.max()
    assert np.max(np.abs(qp[sel] - qa[sel]) / qa[sel]) < 1e-11
