"""The split form's stage kernels against one another where their work splits: the warp rows along
x1 (29 faces each), the walks of 8 faces along x2 and x3, and the one-kernel hydro stage of small
grids, which solves every face from both of its cells with the ghost mapping of single loads.

Two kernels that do the same FP32 arithmetic sit at the same rounding distance from the FP64 form and
apart by rounding noise only: each must be no further from FP64 than 1.5 times the other, and in no cell
may the two differ, or either be off FP64, by more than a bound on that noise.  The bound: an FP32
flux of a flow of Mach number M carries an error of a few 2^-24 M of the cell's own density, pressure,
sound speed, temperature and B^2 in units of the pressure; a step of three stages adds some ten such
errors a face, the few steps here not more than 100 (measured 36 between the forms and FP64, 14 between
two kernels).  A wrong stencil, ghost or face index moves a cell by a fraction of M or of its field, 1e4
times as much and more."""
import numpy as np
import pytest

from phlegethon_b200 import problems
from test_gpu_split import run_form
from util import div_b_max, field_errors, permute_axes

pytestmark = pytest.mark.gpu


def cell_differences(ha, hb):
    """Largest difference in any cell, in units of the cell's density, pressure, sound speed and temperature
    (B of the pressure's root), and the rms Mach number."""
    sd, ip = ha.cfg.sdims, 1 + ha.cfg.sdims
    a, b = ha.interior(ha.prim), hb.interior(hb.prim)
    d, cs = np.abs(a - b), np.sqrt(b[ip] / b[0])
    out = {"rho": (d[0] / b[0]).max(), "p": (d[ip] / b[ip]).max(), "v": (d[1:ip] / cs).max(),
           "e": np.abs(ha.interior(ha.eint) / hb.interior(hb.eint) - 1.0).max(),
           "T": np.abs(ha.interior(ha.temp) / hb.interior(hb.temp) - 1.0).max()}
    if ha.cfg.mhd:
        out["b"] = max(np.abs(ha.bface_interior(k) - hb.bface_interior(k)).max() for k in range(sd)) / np.sqrt(b[ip].min())
    return out, np.sqrt((b[1:ip] ** 2).sum(axis=0).mean()) / cs.mean()


def check(ha, hb, h64):
    ea, eb = field_errors(ha, h64), field_errors(hb, h64)
    for f in ea:
        assert ea[f] <= 1.5 * eb[f] + 1e-12 and eb[f] <= 1.5 * ea[f] + 1e-12, (f, ea, eb)
    for a, b in ((ha, hb), (ha, h64), (hb, h64)):
        diff, mach = cell_differences(a, b)
        for f in diff:
            assert diff[f] <= 100 * 2.0 ** -24 * mach, (f, diff, mach)


def both(cfg, h, table, monkeypatch, var, a, b, steps=3):
    monkeypatch.setenv(var, a)
    ha, sta = run_form(cfg, h, steps, table, "fp32_split")
    monkeypatch.setenv(var, b)
    hb, stb = run_form(cfg, h, steps, table, "fp32_split")
    h64, _ = run_form(cfg, h, steps, table, "fp64")
    for st in (sta, stb):
        assert st["nonfinite"] == 0
        assert st["newton_calls"] == (steps * 3 * cfg.n_cells if cfg.helmholtz else 0)
    check(ha, hb, h64)
    return ha, hb


# row lengths around multiples of 29 faces (nx1 + 1 of them) and walks around multiples of 8
@pytest.mark.parametrize("n,ny,nz", [(4, 4, 5), (27, 7, 8), (28, 8, 7), (29, 9, 16), (57, 15, 5), (58, 16, 4)])
def test_hydro_face_kernels_equal_one_kernel(gpu_lib, table, monkeypatch, n, ny, nz):
    cfg, h = problems.stratified_3d(n, ny=ny, nz=nz, seed=n)
    both(cfg, h, table, monkeypatch, "PHL_STAGE_KERNEL", "faces", "cell")


@pytest.mark.parametrize("perm", [(1, 0, 2), (0, 2, 1)])
def test_hydro_walls_along_x1_and_x3(gpu_lib, table, monkeypatch, perm):
    cfg, h = problems.stratified_3d(10, ny=30, nz=9)
    h = permute_axes(h, perm)
    both(h.cfg, h, table, monkeypatch, "PHL_STAGE_KERNEL", "faces", "cell")


@pytest.mark.parametrize("n", [28, 31, 58])
def test_hydro_2d(gpu_lib, monkeypatch, n):
    cfg, h = problems.hot_bubble_2d(n)
    both(cfg, h, None, monkeypatch, "PHL_STAGE_KERNEL", "faces", "cell", steps=6)


@pytest.mark.parametrize("rec", ["pph", "lim5th"])
def test_hydro_other_reconstructions(gpu_lib, table, monkeypatch, rec):
    cfg, h = problems.stratified_3d(30, ny=9, nz=10, rec=rec)
    both(cfg, h, table, monkeypatch, "PHL_STAGE_KERNEL", "faces", "cell")


@pytest.mark.parametrize("case", ["28", "29", "58", "walls_x1", "walls_x3", "2d"])
def test_mhd_rows_equal_walks(gpu_lib, table, monkeypatch, case):
    if case == "2d":
        cfg, h = problems.orszag_tang_2d(59)
        tab = None
    else:
        cfg, h = problems.stratified_3d(int(case) if case.isdigit() else 12, ny=17, nz=7, mhd=True)
        # a field with all three components: a loop in the (x1, x3) plane adds to the uniform b1
        B = h.b_x[0][0, 0, 0]
        i, k = np.arange(-1, cfg.nx1 + 2), np.arange(-1, cfg.nx3 + 2)
        dx = cfg.dx()
        A = 0.1 * B * cfg.x1u * np.cos(2 * np.pi * i / cfg.nx1)[:, None] * np.cos(2 * np.pi * k / cfg.nx3)[None, :]
        h.b_x[0][...] += ((A[:, 1:] - A[:, :-1]) / dx[2])[:, None, :]
        h.b_x[2][...] += (-(A[1:, :] - A[:-1, :]) / dx[0])[:, None, :]
        tab = table
    if case.startswith("walls"):
        h = permute_axes(h, (1, 0, 2) if case == "walls_x1" else (0, 2, 1))
    ha, hb = both(h.cfg, h, tab, monkeypatch, "PHL_FACE_KERNEL", "row", "walk")
    assert div_b_max(ha) <= 1e-13 and div_b_max(hb) <= 1e-13


@pytest.mark.parametrize("kind", ["cell", "faces"])
@pytest.mark.parametrize("riemann,sdims", [("hllc", 2), ("lhllc", 2), ("hllc", 3), ("hlld", 2)])
def test_a_nan_spreads_as_in_fp64(gpu_lib, monkeypatch, riemann, sdims, kind):
    """One cell with a NaN density: after a step the same cells hold a NaN as in the FP64 form (a NaN
    difference limits the slope to 0, so each stage reaches the neighbouring faces' other cells only).
    The gradients are positive along every axis: both differences at the cells beside the NaN have the
    same sign bit."""
    from phlegethon_b200.abi import Simulation
    from phlegethon_b200.grid import Config, HostGrid
    monkeypatch.setenv("PHL_STAGE_KERNEL", kind)
    n, masks = (17, 16, 18 if sdims == 3 else 1), []
    for form in ("fp64", "fp32_split"):
        cfg = Config(sdims=sdims, nx1=n[0], nx2=n[1], nx3=n[2], ngc=2, nas=0, riemann=riemann, rk_stages=2,
                     mhd=riemann == "hlld", mach_cutoff=1e-4, bc=[["periodic", "periodic"]] * 3, precision=form)
        h = HostGrid(cfg)
        x, y, z = h.coords()
        h.prim[0] = 1.0 + 0.3 * x + 0.4 * y + 0.1 * z
        h.prim[1:1 + sdims] = 0.1
        h.prim[1 + sdims] = 1.0 + 0.2 * x + 0.1 * y + 0.1 * z
        if cfg.mhd:
            for d in range(sdims):
                h.b_x[d][...] = 0.1
        with Simulation(cfg) as sim:
            sim.upload(h)
            sim.init_thermo()
            dt, smax = sim.compute_hyperbolic_dt()
            sim.download(h)
            h.interior(h.prim)[0, 8, 7, n[2] // 2] = np.nan
            sim.upload(h)
            sim.set_time(0.0, dt, smax)
            sim.hydro_step()
            sim.download(h)
        masks.append(np.isnan(h.interior(h.prim)).any(axis=0))
    assert masks[0].any() and np.array_equal(*masks), (masks[0].sum(), masks[1].sum())
