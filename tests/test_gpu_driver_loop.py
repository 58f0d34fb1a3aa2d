"""The driver's per-step calls (hydro_step, compute_hyperbolic_dt) past the point where hydro_step runs as
a graph: the same states bit for bit as the batched loop, with the state re-uploaded, the background
replaced and both buffer parities in between."""
import numpy as np
import pytest

from phlegethon_b200 import problems
from util import max_abs_diff

pytestmark = pytest.mark.gpu


def start(cfg, h, table):
    from phlegethon_b200.abi import Simulation
    sim = Simulation(cfg, table if cfg.helmholtz else None)
    sim.upload(h)
    sim.init_thermo()
    sim.compute_hyperbolic_dt()
    return sim


@pytest.mark.parametrize("case", ["bubble_fp64", "bubble_split", "mhd_split", "orszag_rk2"])
def test_driver_loop_equals_batched_loop(gpu_lib, table, case):
    if case.startswith("bubble"):
        cfg, h = problems.hot_bubble_2d(24)
    elif case == "orszag_rk2":
        cfg, h = problems.orszag_tang_2d(24)
        cfg = cfg.replace(rk_stages=2)
        h.cfg = cfg
    else:
        cfg, h = problems.stratified_3d(12, ny=10, nz=9, mhd=True)
    if case.endswith("split"):
        cfg = cfg.replace(precision="fp32_split")
    n = 23
    ha, hb = h.copy(), h.copy()
    with start(cfg, h, table) as sim:
        for _ in range(n):
            sim.hydro_step()
            dt, smax = sim.compute_hyperbolic_dt()
        sim.download(ha)
    with start(cfg, h, table) as sim:
        for _ in range(n):
            sim.time_loop(1)
            dt2, smax2 = sim.compute_hyperbolic_dt()
        sim.download(hb)
    assert (dt, smax) == (dt2, smax2)
    assert max_abs_diff(ha, hb) == 0.0


def test_new_state_and_background_after_graphs(gpu_lib):
    cfg, h = problems.hot_bubble_2d(20)
    _, h2 = problems.hot_bubble_2d(20)
    h2.prim[1] += 0.01
    h2.phi_cc[...] += 1.0  # another constant in the potential: the energies change with it
    for d in range(2):
        h2.phi_x[d][...] += 1.0
    ha, hb = h2.copy(), h2.copy()
    with start(cfg, h, None) as sim:
        for _ in range(13):
            sim.hydro_step()
            sim.compute_hyperbolic_dt()
        sim.upload(h2)
        sim.init_thermo()
        sim.compute_hyperbolic_dt()
        for _ in range(3):
            sim.hydro_step()
            sim.compute_hyperbolic_dt()
        sim.download(ha)
    with start(cfg, h2, None) as sim:
        for _ in range(3):
            sim.hydro_step()
            sim.compute_hyperbolic_dt()
        sim.download(hb)
    assert max_abs_diff(ha, hb) == 0.0


@pytest.mark.parametrize("precision", ["fp64", "fp32_split"])
def test_full_background_after_a_profile(gpu_lib, precision):
    """The first background is a profile along x2, the second varies along x1: its arrays are larger, and
    the step graphs hold the layout and the addresses of the first.  Same states as a fresh context."""
    cfg, h = problems.hot_bubble_2d(20)
    cfg = cfg.replace(precision=precision)
    h2 = h.copy()
    x = h.coords()[0]
    wave = lambda x: 1.0 + 1e-3 * np.sin(2.0 * np.pi * x)
    h2.eq_prim_cc[:2] *= wave(x)
    for d in range(2):
        h2.eq_prim_x[d][:2] *= wave(h.face_coords(d)[0])
    ha, hb, hc = h2.copy(), h2.copy(), h.copy()

    def steps(sim):
        for _ in range(3):
            sim.hydro_step()
            sim.compute_hyperbolic_dt()
        sim.time_loop(3)

    def again(sim, h):
        sim.upload(h)
        sim.init_thermo()
        sim.compute_hyperbolic_dt()

    with start(cfg, h, None) as sim:
        for _ in range(13):
            sim.hydro_step()
            sim.compute_hyperbolic_dt()
        sim.time_loop(2)
        again(sim, h2)
        steps(sim)
        sim.download(ha)
        again(sim, h)  # and the profile again
        steps(sim)
        sim.download(hc)
    with start(cfg, h2, None) as sim:
        steps(sim)
        sim.download(hb)
    assert np.isfinite(hb.interior(hb.prim)).all()
    assert max_abs_diff(ha, hb) == 0.0
    hd = h.copy()
    with start(cfg, h, None) as sim:
        if cfg.precision == "fp32_split":
            # the scales of the split form are those of the first state a context was given
            assert h.prim[0].max() == h2.prim[0].max() and h.prim[3].max() == h2.prim[3].max()
        steps(sim)
        sim.download(hd)
    assert max_abs_diff(hc, hd) == 0.0


def test_tmax_and_steps_between_calls(gpu_lib):
    """steps_done and the time of consecutive calls, with the clamp to tmax and calls that do nothing."""
    cfg, h = problems.hot_bubble_2d(16)
    with start(cfg, h, None) as sim:
        done, t1 = sim.time_loop(3)
        assert done == 3
        done, t2 = sim.time_loop(0)
        assert done == 0 and t2 == t1
        done, t3 = sim.time_loop(50, t1 * 2.5)
        assert 0 < done < 50 and t3 == t1 * 2.5
        done, t4 = sim.time_loop(4, t3)
        assert done == 0 and t4 == t3
        done, t5 = sim.time_loop(1)
        assert done == 1 and t5 > t4
        assert sim.status()["steps"] > 4
