"""What the host does with device memory, on the CPU: the library linked with a runtime that has no device
(hostrt.py)."""
import numpy as np
import pytest

import hostrt
from phlegethon_b200 import problems


@pytest.fixture(scope="module")
def host_lib(tmp_path_factory):
    return hostrt.link(tmp_path_factory.mktemp("hostrt"))


@pytest.fixture
def rt(host_lib, monkeypatch):
    from phlegethon_b200 import abi
    monkeypatch.setattr(abi, "_lib", None)
    abi.load_library(host_lib)
    fake = hostrt.FakeRuntime(host_lib)
    fake.reset()
    fake.clear_watches()
    yield fake
    fake.reset()


def tiny_table(cfg):
    """A table of the configuration's size whose values no kernel reads here."""
    return np.zeros((9, cfg.helm_nrho, cfg.helm_nT)), np.zeros((4, cfg.helm_nrho, cfg.helm_nT))


def started(cfg, h):
    from phlegethon_b200.abi import Simulation
    sim = Simulation(cfg, tiny_table(cfg) if cfg.helmholtz else None)
    sim.upload(h)
    sim.init_thermo()
    sim.compute_hyperbolic_dt()
    return sim


def uneven(h):
    """A background that is no profile along x2 any more (what the host checks is its layout)."""
    h = h.copy()
    h.eq_prim_cc[0] *= 1.0 + 1e-3 * np.arange(h.eq_prim_cc.shape[1])[:, None, None]
    return h


def problem(case):
    if case == "bubble":
        cfg, h = problems.hot_bubble_2d(12, shock_flattening=False)
    else:
        cfg, h = problems.stratified_3d(6, ny=10, nz=5, mhd=case == "mhd")
    return cfg, h


def k_unpack_fits(rt):
    """Every k_unpack launch writes its n cells times ncomp components inside a live block."""
    rows = rt.launches_of("k_unpack")
    for _, (_, _, _, n0, n1, n2, _, _, _, _, _, ncomp, stride), room in rows:
        assert room[1] >= 8 * (n0 * n1 * n2 + (ncomp - 1) * stride), (n0, n1, n2, ncomp, room[1])
    return len(rows)


def k_scale_fits(rt):
    rows = rt.launches_of("k_scale_f32")
    for _, (_, _, n, _), room in rows:
        assert room[0] >= 8 * n and room[1] >= 4 * (4 * (n - 1) + 1), (n, room)
    return len(rows)


# ------------------------------------------------------------------ background
@pytest.mark.parametrize("precision", ["fp64", "fp32_split"])
@pytest.mark.parametrize("case", ["bubble", "hydro", "mhd"])
def test_background_buffers_grow_with_the_layout(rt, case, precision):
    """A context whose first background was a profile takes a full one later (and a profile again): every
    array the kernels write holds what they write."""
    cfg, h = problem(case)
    cfg = cfg.replace(precision=precision)
    rt.watch("k_unpack", "PPiiiiiiiiiiP")
    rt.watch("k_scale_f32", "PPPP")
    with started(cfg, h) as sim:
        before = rt.launches_of("k_unpack")
        sim.upload(uneven(h))
        assert k_unpack_fits(rt) > len(before)
        assert (k_scale_fits(rt) > 0) == (precision == "fp32_split")
        sim.time_loop(2)
        sim.upload(h)
        k_unpack_fits(rt)
        k_scale_fits(rt)
    assert rt.violations() == 0


def test_refused_background_leaves_a_context_that_does_not_run(rt):
    """An upload that finds no room for a full background fails, the steps are refused until another
    upload succeeds, and no graph of the old layout is left."""
    from phlegethon_b200.abi import PhlError
    cfg, h = problem("hydro")
    cfg = cfg.replace(precision="fp32_split")
    rt.watch("k_unpack", "PPiiiiiiiiiiP")
    rt.watch("k_scale_f32", "PPPP")
    full, refused = uneven(h), 0
    with started(cfg, h) as sim:
        sim.time_loop(2)
        for k in range(100):
            rt.refuse(k)
            try:
                sim.upload(full)
                rt.refuse(-1)
                break
            except PhlError as e:
                assert e.code == -2
                refused += 1
            rt.refuse(-1)
            for call in (lambda: sim.time_loop(1), sim.hydro_step):
                with pytest.raises(PhlError) as e:
                    call()
                assert e.value.code == -4
            sim.upload(h)  # a profile again: runs
            sim.time_loop(1)
        k_unpack_fits(rt)
        k_scale_fits(rt)
        assert refused > 0
        sim.time_loop(1)
    assert rt.violations() == 0
