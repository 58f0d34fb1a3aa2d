"""FP32 split-precision form against the FP64 form (and the FP64 oracle).

The split form keeps the conserved state in FP64 and computes fluxes in FP32 on well-balanced
deviations, so its results are not bitwise equal to FP64; the bar is the per-field relative L1
error the split form is built for (density <= 1e-5 after 1000 steps of the 256^3 box).  The
limits here sit 5-20x above the errors measured on the B200 for each case (FP32 rounding moves
with code generation; a real regression moves them by orders of magnitude).
"""
import numpy as np
import pytest

from phlegethon_b200 import problems
from util import field_errors

pytestmark = pytest.mark.gpu


def run_form(cfg, h, nsteps, table, precision):
    from phlegethon_b200.abi import Simulation
    c = cfg.replace(precision=precision)
    hg = h.copy()
    with Simulation(c, table if c.helmholtz else None) as sim:
        sim.upload(hg)
        sim.init_thermo()
        sim.compute_hyperbolic_dt()
        done, _ = sim.time_loop(nsteps)
        assert done == nsteps
        sim.download(hg)
        st = sim.status()
    return hg, st


@pytest.mark.parametrize("riemann", ["lhllc", "hllc"])
def test_split_stratified_helmholtz(gpu_lib, oracle, table, riemann):
    cfg, h = problems.stratified_3d(16, ny=24, nz=12, riemann=riemann)
    h64, _ = run_form(cfg, h, 40, table, "fp64")
    h32, st = run_form(cfg, h, 40, table, "fp32_split")
    err = field_errors(h32, h64)
    assert st["nonfinite"] == 0 and st["newton_nonconverged"] == 0
    # measured after 40 steps: LHLLC rho 2e-10, T 5e-10, v <= 1.8e-7; HLLC (dissipative at
    # Mach 1e-3, see MHD_LIMITS) rho 1.3e-7, T 3.2e-7, v <= 1.2e-4
    thermo, vlim = (1e-8, 1e-6) if riemann == "lhllc" else (1e-6, 5e-4)
    assert err["rho"] <= thermo, err
    assert err["p"] <= thermo, err
    assert err["T"] <= thermo, err
    for d in (1, 2, 3):
        assert err["v%d" % d] <= vlim, err


def test_split_hot_bubble(gpu_lib, oracle):
    cfg, h = problems.hot_bubble_2d(64)
    h64, _ = run_form(cfg, h, 60, None, "fp64")
    h32, _ = run_form(cfg, h, 60, None, "fp32_split")
    err = field_errors(h32, h64)
    # measured after 60 steps: rho 1.9e-10, p 1e-10, v <= 8.6e-8
    assert err["rho"] <= 1e-8, err
    assert err["p"] <= 1e-8, err
    assert err["v1"] <= 1e-6 and err["v2"] <= 1e-6, err


def test_split_keeps_hydrostatic_balance(gpu_lib, table):
    cfg, h = problems.stratified_3d(12, ny=16, nz=10, mach=0.0)
    h32, st = run_form(cfg, h, 20, table, "fp32_split")
    v = np.abs(h32.interior(h32.prim)[1:4]).max()
    cs = np.sqrt(5.0 / 3.0 * h32.interior(h32.prim)[4] / h32.interior(h32.prim)[0]).min()
    assert v / cs < 1e-9


@pytest.mark.parametrize("riemann", ["lhllc", "hllc"])
def test_face_kernels_equal_one_kernel_stage(gpu_lib, table, riemann, monkeypatch):
    """The hydro stage through the face kernels against the one-kernel stage, which solves every face
    twice (once per neighbour, so its two copies of a face flux can differ in the last FP32 bits where
    the compiler contracts differently).  Both sit at the same FP32 rounding distance from the FP64
    form."""
    cfg, h = problems.stratified_3d(32, ny=16, nz=32, riemann=riemann)
    monkeypatch.setenv("PHL_STAGE_KERNEL", "cell")
    hc, stc = run_form(cfg, h, 6, table, "fp32_split")
    monkeypatch.setenv("PHL_STAGE_KERNEL", "faces")
    hf, stf = run_form(cfg, h, 6, table, "fp32_split")
    h64, _ = run_form(cfg, h, 6, table, "fp64")
    assert stf["nonfinite"] == 0 and stf["newton_nonconverged"] == 0
    e_f = field_errors(hf, h64)
    e_c = field_errors(hc, h64)
    diff = field_errors(hf, hc)
    for f in e_c:
        # no further from FP64 than the one-kernel stage, and apart by FP32 rounding noise only
        assert e_f[f] <= 1.5 * e_c[f] + 1e-12, (f, e_f, e_c)
        assert diff[f] <= 2.0 * e_c[f] + 1e-12, (f, diff, e_c)


@pytest.mark.parametrize("n,ny,nz,kind", [(96, 24, 32, "cell"), (64, 64, 64, "faces")])
def test_default_stage_is_the_one_its_size_selects(gpu_lib, table, monkeypatch, n, ny, nz, kind):
    """A grid below and one above the one-kernel line: the default run is the selected form's, bit for
    bit."""
    cfg, h = problems.stratified_3d(n, ny=ny, nz=nz)
    monkeypatch.setenv("PHL_STAGE_KERNEL", kind)
    ha, sta = run_form(cfg, h, 4, table, "fp32_split")
    monkeypatch.delenv("PHL_STAGE_KERNEL")
    hb, stb = run_form(cfg, h, 4, table, "fp32_split")
    assert stb["nonfinite"] == 0 and stb["tensor_core_stalls"] == 0
    assert stb["newton_iterations"] == sta["newton_iterations"]
    for a, b in ((ha.prim, hb.prim), (ha.temp, hb.temp), (ha.eint, hb.eint)):
        assert np.array_equal(ha.interior(a), hb.interior(b))


# ------------------------------------------------------------------------------ MHD
@pytest.mark.parametrize("riemann", ["hlld", "lhlld"])
def test_split_orszag_tang(gpu_lib, riemann):
    """Split MHD (FP32 HLLD/LHLLD, FP32 EMFs, FP64 face-B update) against the FP64 form."""
    from util import div_b_max
    cfg, h = problems.orszag_tang_2d(64, riemann=riemann)
    h64, _ = run_form(cfg, h, 30, None, "fp64")
    h32, st = run_form(cfg, h, 30, None, "fp32_split")
    err = field_errors(h32, h64)
    assert st["nonfinite"] == 0
    # measured <= 1e-7 in every field (Orszag-Tang variants, 30 steps)
    for f in ("rho", "p", "e", "v1", "v2", "b1", "b2"):
        assert err[f] <= 5e-7, (f, err)
    assert div_b_max(h32) <= 1e-13


# LHLLD (the low-dissipation solver the low-Mach box is run with) keeps FP32 rounding-level
# errors; HLLD's dissipative flux f + s (U* - U) cancels O(Mach) differences of O(1) states, so
# its FP32 velocity and induction fluxes carry relative errors ~ eps / Mach
MHD_LIMITS = {"lhlld": {"thermo": 1e-8, "v": 1e-6, "b": 1e-6},   # measured 3.6e-10, 1.2e-7, 5.7e-8
              "hlld": {"thermo": 1e-6, "v": 5e-4, "b": 1e-3}}    # measured 2.9e-7, 1.1e-4, 2e-4


@pytest.mark.parametrize("riemann", ["lhlld", "hlld"])
def test_split_stratified_helmholtz_mhd(gpu_lib, table, riemann):
    from util import div_b_max
    cfg, h = problems.stratified_3d(16, ny=24, nz=12, mhd=True, riemann=riemann)
    h64, _ = run_form(cfg, h, 30, table, "fp64")
    h32, st = run_form(cfg, h, 30, table, "fp32_split")
    err = field_errors(h32, h64)
    lim = MHD_LIMITS[riemann]
    assert st["nonfinite"] == 0 and st["newton_nonconverged"] == 0
    for f in ("rho", "p", "e", "T"):
        assert err[f] <= lim["thermo"], (f, err)
    for f in ("v1", "v2", "v3"):
        assert err[f] <= lim["v"], (f, err)
    for f in ("b1", "b2", "b3"):
        assert err[f] <= lim["b"], (f, err)
    assert div_b_max(h32) <= 1e-13


@pytest.mark.parametrize("mhd,riemann", [(False, "lhllc"), (True, "lhlld")])
def test_split_helmholtz_without_fasteos(gpu_lib, table, mhd, riemann):
    """Split form of the Helmholtz path without FASTEOS: helm_rhoP_given (FP64) per Riemann side
    from the FP32 face state, tiled and per-cell grids."""
    for n, ny, nz in ((16, 24, 12), (32, 16, 16)):
        cfg, h = problems.stratified_3d(n, ny=ny, nz=nz, mhd=mhd, riemann=riemann, fasteos=False)
        h64, _ = run_form(cfg, h, 20, table, "fp64")
        h32, st = run_form(cfg, h, 20, table, "fp32_split")
        err = field_errors(h32, h64)
        assert st["nonfinite"] == 0 and st["newton_nonconverged"] == 0
        # measured: rho, p, e, T <= 2.3e-10, v <= 8.5e-8
        for f in ("rho", "p", "e", "T"):
            assert err[f] <= 1e-8, (f, err)
        for f in ("v1", "v2", "v3"):
            assert err[f] <= 1e-6, (f, err)


def test_split_orszag_tang_lim5th(gpu_lib):
    from util import div_b_max
    cfg, h = problems.orszag_tang_2d(64, rec="lim5th")
    h64, _ = run_form(cfg, h, 30, None, "fp64")
    h32, st = run_form(cfg, h, 30, None, "fp32_split")
    err = field_errors(h32, h64)
    assert st["nonfinite"] == 0
    # measured <= 1e-7 in every field (Orszag-Tang variants, 30 steps)
    for f in ("rho", "p", "e", "v1", "v2", "b1", "b2"):
        assert err[f] <= 5e-7, (f, err)
    assert div_b_max(h32) <= 1e-13


@pytest.mark.parametrize("mhd,riemann,rec,dims", [(True, "lhlld", "pph", (16, 24, 12)), (True, "lhlld", "lim5th", (16, 24, 12)),
                                                  (False, "lhllc", "pph", (32, 16, 16)),
                                                  (False, "lhllc", "lim5th", (32, 16, 16))])
def test_split_stratified_higher_order(gpu_lib, table, mhd, riemann, rec, dims):
    n, ny, nz = dims
    cfg, h = problems.stratified_3d(n, ny=ny, nz=nz, mhd=mhd, riemann=riemann, rec=rec)
    h64, _ = run_form(cfg, h, 20, table, "fp64")
    h32, st = run_form(cfg, h, 20, table, "fp32_split")
    err = field_errors(h32, h64)
    assert st["nonfinite"] == 0 and st["newton_nonconverged"] == 0
    # measured: thermodynamic fields <= 3.4e-10, v <= 1.1e-7
    for f in ("rho", "p", "e", "T"):
        assert err[f] <= 1e-8, (f, err)
    for f in ("v1", "v2", "v3"):
        assert err[f] <= 1e-6, (f, err)


@pytest.mark.parametrize("mhd,riemann", [(False, "lhllc"), (True, "lhlld")])
def test_split_on_fermi_table(gpu_lib, mhd, riemann):
    """The split form on the electron-positron Fermi-gas table against FP64."""
    from phlegethon_b200 import helm_fermi
    from test_helm_fermi import SMALL
    table = helm_fermi.generate(**SMALL)
    cfg, h = problems.stratified_3d(16, ny=24, nz=12, mhd=mhd, riemann=riemann, table=dict(SMALL), eos_model="fermi")
    h64, _ = run_form(cfg, h, 20, table, "fp64")
    h32, st = run_form(cfg, h, 20, table, "fp32_split")
    err = field_errors(h32, h64)
    assert st["nonfinite"] == 0 and st["newton_nonconverged"] == 0
    assert err["rho"] <= 1e-8 and err["p"] <= 1e-8 and err["T"] <= 1e-8, err  # measured <= 2.8e-10


# ------------------------------------------------------------------------------ USE_SHOCK_FLATTENING
def test_split_blast_shock_flattening(gpu_lib):
    """Detector on the FP32 state, PLM fallback and HLL faces, against the FP64 form."""
    cfg, h = problems.blast_2d(64, riemann="hllc")
    h64, _ = run_form(cfg, h, 20, None, "fp64")
    h32, st = run_form(cfg, h, 20, None, "fp32_split")
    err = field_errors(h32, h64)
    assert st["nonfinite"] == 0
    for f in ("rho", "p", "e"):
        assert err[f] <= 5e-7, (f, err)  # measured rho 3.4e-9, p and e 4.1e-8


def test_split_orszag_tang_shock_flattening(gpu_lib):
    from util import div_b_max
    cfg, h = problems.orszag_tang_2d(64, riemann="hlld", shock_flattening=True)
    h64, _ = run_form(cfg, h, 30, None, "fp64")
    h32, st = run_form(cfg, h, 30, None, "fp32_split")
    err = field_errors(h32, h64)
    assert st["nonfinite"] == 0
    # measured <= 1e-7 in every field (Orszag-Tang variants, 30 steps)
    for f in ("rho", "p", "e", "v1", "v2", "b1", "b2"):
        assert err[f] <= 5e-7, (f, err)
    assert div_b_max(h32) <= 1e-13


@pytest.mark.parametrize("mhd,rec", [(False, "lim2nd"), (False, "pph"), (True, "lim2nd")])
def test_split_stratified_shock_flattening(gpu_lib, table, mhd, rec):
    """eps_sf = 0.4 flags the upper part of the box; with WB and FASTEOS this includes the x1
    sweep's gamma_e handling on flagged faces."""
    cfg, h = problems.stratified_3d(16, ny=16, nz=12, mhd=mhd, rec=rec, shock_flattening=True, eps_sf=0.4)
    h64, _ = run_form(cfg, h, 20, table, "fp64")
    h32, st = run_form(cfg, h, 20, table, "fp32_split")
    err = field_errors(h32, h64)
    assert st["nonfinite"] == 0 and st["newton_nonconverged"] == 0
    for f in ("rho", "p", "e", "T"):
        assert err[f] <= 2e-7, (f, err)  # measured <= 2.6e-8


def test_split_all_mach_orszag_tang(gpu_lib):
    """FLUX_IS_ALL_MACH in the FP32 LHLLD against the FP64 form."""
    cfg, h = problems.orszag_tang_2d(64, riemann="lhlld")
    h.cfg = cfg = cfg.replace(all_mach=True)
    h64, _ = run_form(cfg, h, 30, None, "fp64")
    h32, st = run_form(cfg, h, 30, None, "fp32_split")
    err = field_errors(h32, h64)
    assert st["nonfinite"] == 0
    # measured <= 1e-7 in every field (Orszag-Tang variants, 30 steps)
    for f in ("rho", "p", "e", "v1", "v2", "b1", "b2"):
        assert err[f] <= 5e-7, (f, err)


@pytest.mark.parametrize("mhd", [False, True])
def test_split_constant_acceleration(gpu_lib, table, mhd):
    """USE_CONSTANT_ACCELERATION in the split form's FP64 update against the FP64 form."""
    cfg, h = problems.stratified_3d(16, ny=16, nz=16, mhd=mhd)
    h.cfg = cfg = cfg.replace(constant_acceleration=True, acc=(3.0e5, 0.0, -2.0e5))
    h64, _ = run_form(cfg, h, 20, table, "fp64")
    h32, st = run_form(cfg, h, 20, table, "fp32_split")
    err = field_errors(h32, h64)
    assert st["nonfinite"] == 0 and st["newton_nonconverged"] == 0
    # measured: thermodynamic fields <= 3e-10, v <= 1e-7
    for f in ("rho", "p", "e", "T"):
        assert err[f] <= 1e-8, (f, err)
    for f in ("v1", "v3"):
        assert err[f] <= 1e-6, (f, err)


# ------------------------------------------------------------------------------ split against the oracle
def _oracle_run(oracle, cfg, h, nsteps, table):
    ho = h.copy()
    helm = oracle.Helm.for_config(cfg, *table) if cfg.helmholtz else None
    o = oracle.OracleGrid(ho, helm)
    o.init_thermo()
    o.compute_hyperbolic_dt()
    o.time_loop(nsteps)
    return ho


# per family: (maker, steps, {field group: limit}); the limits sit a few times above the errors
# measured on the B200 for these cases
ORACLE_CASES = {
    "hot_bubble": (lambda: problems.hot_bubble_2d(48), 20, {"thermo": 1e-9, "v": 1e-6}),
    "orszag_tang_lhlld": (lambda: problems.orszag_tang_2d(48, riemann="lhlld"), 20, {"thermo": 5e-7, "v": 5e-7, "b": 5e-7}),
    "stratified": (lambda: problems.stratified_3d(12, ny=16, nz=10), 10, {"thermo": 1e-8, "v": 5e-7}),
    "stratified_mhd": (lambda: problems.stratified_3d(12, ny=16, nz=10, mhd=True), 10,
                       {"thermo": 1e-8, "v": 5e-7, "b": 1e-6}),
}


@pytest.mark.parametrize("family", sorted(ORACLE_CASES))
def test_split_against_oracle(gpu_lib, oracle, table, family):
    """The split form directly against the CPU oracle (not through the FP64 GPU form)."""
    maker, nsteps, lim = ORACLE_CASES[family]
    cfg, h = maker()
    tab = table if cfg.helmholtz else None
    ho = _oracle_run(oracle, cfg, h, nsteps, tab)
    h32, st = run_form(cfg, h, nsteps, tab, "fp32_split")
    err = field_errors(h32, ho)
    assert st["nonfinite"] == 0
    groups = {"thermo": ("rho", "p", "e", "T"), "v": ("v1", "v2", "v3"), "b": ("b1", "b2", "b3")}
    for grp, limit in lim.items():
        for f in groups[grp]:
            if f in err:
                assert err[f] <= limit, (f, err)


@pytest.mark.parametrize("mhd_case", ["stratified_mhd", "orszag_tang"])
def test_row_faces_equal_walking_faces(gpu_lib, table, mhd_case, monkeypatch):
    """The x1 faces by warp rows (the default) against the walking face kernel along x1: the same edges
    and the same solver on the same inputs, so both sit at the same FP32 rounding distance from the FP64
    form and apart by rounding noise only (the compiler contracts the edge arithmetic differently in the
    two kernels)."""
    if mhd_case == "stratified_mhd":
        cfg, h = problems.stratified_3d(128, ny=16, nz=8, mhd=True)
        tab = table
    else:
        cfg, h = problems.orszag_tang_2d(256)
        tab = None
    monkeypatch.setenv("PHL_FACE_KERNEL", "walk")
    ha, sta = run_form(cfg, h, 3, tab, "fp32_split")
    monkeypatch.setenv("PHL_FACE_KERNEL", "row")
    hb, stb = run_form(cfg, h, 3, tab, "fp32_split")
    h64, _ = run_form(cfg, h, 3, tab, "fp64")
    assert stb["nonfinite"] == 0 and stb["tensor_core_stalls"] == 0
    e_w = field_errors(ha, h64)
    e_t = field_errors(hb, h64)
    diff = field_errors(hb, ha)
    for f in e_w:
        assert e_t[f] <= 1.5 * e_w[f] + 1e-13, (f, e_t, e_w)
        assert diff[f] <= 2.0 * e_w[f] + 1e-13, (f, diff, e_w)
