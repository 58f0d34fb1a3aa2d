"""What the host does with device memory, on the CPU: the library linked with a runtime that has no device
(hostrt.py)."""
import ctypes as C
import gc

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
    assert rt.violations() == 0 and rt.used() == 0


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
    assert rt.violations() == 0 and rt.used() == 0


# ------------------------------------------------------------------ buffers that could not be replaced
PSTRIDE, TILE = 4608, 64  # floats per partial gradient, samples per block of k_mlp_train_step


def train_launches_fit(rt):
    """Every training launch finds its samples, partial gradients and losses in live blocks."""
    rows = rt.launches_of("k_mlp_train_step")
    for grid, (_, _, _, _, n, _, batch, _, _), room in rows:
        assert room[0] > 0 and room[1] > 0
        assert room[2] >= 16 * n and room[3] >= 4 * n
        assert room[7] >= 4 * PSTRIDE * grid and room[8] >= 4 * batch and grid * TILE == batch
    for _, _, room in rt.launches_of("k_mlp_adam") + rt.launches_of("k_mlp_reduce"):
        assert all(room[i] > 0 for i in (0, 2))
    return len(rows)


def each_refusal(rt, call, retry):
    """call() with its first, second, ... allocation refused, retry() after each; the number refused."""
    refused = 0
    while True:
        rt.refuse(refused)
        rc = call()
        rt.refuse(-1)
        if rc == 0:
            return refused
        assert rc == -2 and refused < 30
        refused += 1
        retry()


def test_training_after_a_refused_allocation(rt):
    """Training and gradient calls whose buffers could not grow, then calls of the old sizes."""
    cfg, h = problem("hydro")
    rt.watch("k_mlp_train_step", "PPPPPPiPP")
    rt.watch("k_mlp_adam", "PiPPP")
    rt.watch("k_mlp_reduce", "PiP")
    feat, target, grad = np.zeros((4096, 4), np.float32), np.zeros(4096, np.float32), np.zeros(4545, np.float32)
    with started(cfg, h) as sim:
        loss = C.c_double()
        train = lambda n, batch: sim.lib.phl_mlp_train(sim.ctx, n, 1, 1, batch, 1e-3, C.byref(loss))
        gradient = lambda n: sim.lib.phl_mlp_gradient(sim.ctx, n, feat.ctypes.data, target.ctypes.data,
                                                      grad.ctypes.data, C.byref(loss))

        def again(n, batch):
            assert train(n, batch) == 0 and gradient(batch) == 0

        # the first call of a context, parameters included
        assert each_refusal(rt, lambda: train(256, 64), lambda: None) > 1
        # more samples, a larger batch, gradients of more samples than a batch
        assert each_refusal(rt, lambda: train(2048, 64), lambda: again(256, 64)) > 0
        assert each_refusal(rt, lambda: train(2048, 512), lambda: again(2048, 64)) > 0
        assert each_refusal(rt, lambda: gradient(4096), lambda: again(2048, 512)) > 0
        again(256, 64)
        assert train_launches_fit(rt) > 40
    assert rt.violations() == 0 and rt.used() == 0


@pytest.mark.parametrize("guess", [0, 1, 2])
def test_batch_after_a_refused_allocation(rt, guess):
    """Batch inversions of host arrays whose buffers could not grow, then smaller ones."""
    cfg, h = problem("hydro")
    rt.watch("k_eos_guess", "ssPPPPPPPP")
    kernel = "k_eos_invertILi%dE" % guess
    rt.watch(kernel, "sPPPPPPPPPPPP")
    with started(cfg, h) as sim:
        assert sim.lib.phl_mlp_set_params(sim.ctx, (C.c_float * 4545)()) == 0

        def invert(n):
            a = [np.ones(n) for _ in range(7)]
            it = np.zeros(n, np.int32)
            return sim.lib.phl_eos_invert_batch(sim.ctx, n, *[x.ctypes.data for x in a], it.ctypes.data, guess)
        assert each_refusal(rt, lambda: invert(100), lambda: None) > 0
        assert each_refusal(rt, lambda: invert(1000), lambda: invert(50)) > 0
        for _, (_, n, *_), room in rt.launches_of(kernel):
            assert all(room[i] >= 8 * n for i in range(2, 9)) and room[9] >= 4 * n
            if guess == 1:
                assert room[10] >= 4 * n and room[12] >= 8 * (n + 1)
        if guess == 1:
            for _, (_, _, _, n, *_), room in rt.launches_of("k_eos_guess"):
                assert room[8] >= 4 * n
    assert rt.violations() == 0 and rt.used() == 0


@pytest.mark.parametrize("case", ["bubble", "hydro", "mhd"])
def test_calls_after_a_refused_allocation(rt, case):
    """The table, the upload and the host pipeline with each of their allocations refused in turn: the call
    fails and succeeds when it is made again, and nothing is left when the context goes."""
    from phlegethon_b200.abi import Simulation, PhlError
    cfg, h = problem(case)
    cfg = cfg.replace(precision="fp32_split")
    rt.watch("k_unpack", "PPiiiiiiiiiiP")

    def code(call):
        try:
            call()
            return 0
        except PhlError as e:
            return e.code
    k = 0
    while True:  # contexts whose initialisation is refused leave nothing behind
        rt.refuse(k)
        try:
            sim = Simulation(cfg, tiny_table(cfg) if cfg.helmholtz else None)
            break
        except PhlError as e:
            assert e.code == -2 and k < 100
        rt.refuse(-1)
        gc.collect()
        k += 1
    rt.refuse(-1)
    with sim:
        if cfg.helmholtz:
            assert each_refusal(rt, lambda: code(lambda: sim.load_helm_table(*tiny_table(cfg))), lambda: None) == 0
        assert each_refusal(rt, lambda: code(lambda: sim.upload(h)), lambda: None) > 0
        sim.init_thermo()
        sim.compute_hyperbolic_dt()
        assert each_refusal(rt, lambda: code(lambda: sim.time_loop_host_async(h, 1)), sim.wait_host) > 0
        sim.wait_host()
        sim.time_loop(1)
        sim.download(h.copy())
        k_unpack_fits(rt)
    assert rt.violations() == 0 and rt.used() == 0


# ------------------------------------------------------------------ face fluxes of the split hydro form
def hydro_calls(cfg, h):
    """Every call of a context that allocates, and steps before and after."""
    with started(cfg, h) as sim:
        sim.time_loop(2)
        sim.time_loop_host_async(h.copy(), 1)
        sim.wait_host()
        for _ in range(12):
            sim.hydro_step()
            sim.compute_hyperbolic_dt()
        n = 64
        a = [np.ones(n) for _ in range(7)]
        if cfg.helmholtz:
            assert sim.lib.phl_mlp_train(sim.ctx, 256, 1, 1, 64, 1e-3, None) == 0
            assert sim.lib.phl_eos_invert_batch(sim.ctx, n, *[x.ctypes.data for x in a], None, 1) == 0
        sim.time_loop(2)
        sim.download(h.copy())


def faces(cfg):
    return [cfg.n_cells // n * (n + 1) for n in (cfg.nx1, cfg.nx2, cfg.nx3)[:cfg.sdims]]


def stage_kernels(rt):
    return {k: len(rt.launches_of(k)) for k in ("k_stage_split", "k_face_split")}


def watch_stages(rt):
    rt.watch("k_stage_split", "s")
    rt.watch("k_face_split", "s")  # walks and rows as well


@pytest.mark.parametrize("case", ["bubble", "hydro"])
def test_no_call_fails_for_the_face_fluxes(rt, monkeypatch, case):
    """A domain runs on a device that has room for it without the face fluxes, whether they fit at first or
    not: they are given back when another allocation finds no room."""
    cfg, h = problem(case)
    cfg = cfg.replace(precision="fp32_split")
    monkeypatch.setenv("PHL_STAGE_KERNEL", "faces")
    hydro_calls(cfg, h)
    with_fluxes = rt.peak()
    without = with_fluxes - sum(4 * ((cfg.nvars * n + 63) // 64 * 64) for n in faces(cfg))
    watch_stages(rt)
    kinds = set()
    for room in np.linspace(without, with_fluxes, 9).astype(int):
        rt.reset()
        rt.room(int(room))
        hydro_calls(cfg, h)
        assert rt.violations() == 0 and rt.used() == 0
        n = stage_kernels(rt)
        kinds.add((n["k_stage_split"] > 0, n["k_face_split"] > 0))
    # room until a later call, room to the end
    assert kinds == {(True, True), (False, True)}


def test_refused_face_fluxes(rt, monkeypatch):
    """phl_init with each allocation refused: fails, or (the face fluxes, or one after them) goes on without."""
    from phlegethon_b200.abi import PhlError, Simulation
    cfg, h = problem("bubble")
    cfg = cfg.replace(precision="fp32_split")
    monkeypatch.setenv("PHL_STAGE_KERNEL", "faces")
    watch_stages(rt)
    went_on = 0
    for k in range(40):
        rt.reset()
        rt.refuse(k)
        try:
            sim = Simulation(cfg)
        except PhlError as e:
            assert e.code == -2
            continue
        refused = rt.mallocs() > k
        rt.refuse(-1)
        with sim:
            sim.upload(h)
            sim.init_thermo()
            sim.compute_hyperbolic_dt()
            sim.time_loop(1)
        n = stage_kernels(rt)
        assert (n["k_stage_split"] > 0) == refused and (n["k_face_split"] > 0) == (not refused)
        went_on += refused
        if not refused:
            break
    assert went_on > 1


def test_small_grids_hold_no_face_fluxes(rt, monkeypatch):
    """A grid whose hydro stages run in one kernel has no use for the face fluxes."""
    cfg, h = problem("hydro")
    cfg = cfg.replace(precision="fp32_split")
    used = {}
    for kind in ("auto", "cell", "faces"):
        monkeypatch.setenv("PHL_STAGE_KERNEL", kind)
        with started(cfg, h):
            used[kind] = rt.used()
    assert used["auto"] == used["cell"]
    assert used["faces"] >= used["cell"] + 4 * cfg.nvars * sum(faces(cfg))


@pytest.mark.parametrize("case,below,above", [("bubble", 237, 239), ("lim2nd", 38, 39), ("pph", 38, 39),
                                              ("lim5th", 26, 27), ("sf", 38, 39), ("sf_pph", 26, 27), ("given", 38, 39)])
def test_one_kernel_line_is_in_waves(rt, case, below, above):
    """Hydro stages run in one kernel up to three waves of its blocks (one for LIM5TH and flattened PPH): here of
    one block of 128 cells on each of 148 SMs."""
    waves = 1 if case in ("lim5th", "sf_pph") else 3
    watch_stages(rt)
    for n in (below, above):
        if case == "bubble":
            cfg, h = problems.hot_bubble_2d(n)
        else:
            cfg, h = problems.stratified_3d(n, rec=case[-3:] if "pph" in case else case if case == "lim5th" else "lim2nd",
                                            shock_flattening=case.startswith("sf"), fasteos=case != "given")
        assert (cfg.n_cells <= waves * 148 * 128) == (n == below)
        rt.reset()
        rt.blocks_per_sm(1)
        with started(cfg.replace(precision="fp32_split"), h) as sim:
            sim.time_loop(1)
        k = stage_kernels(rt)
        assert (k["k_stage_split"] > 0, k["k_face_split"] > 0) == (n == below, n == above), n


def test_refused_graph_gives_the_face_fluxes_back(rt, monkeypatch):
    """No room for a step graph: the face fluxes make some."""
    cfg, h = problem("hydro")
    monkeypatch.setenv("PHL_STAGE_KERNEL", "faces")
    watch_stages(rt)
    with started(cfg.replace(precision="fp32_split"), h) as sim:
        before = rt.used()
        rt.refuse_graphs(1)  # the next one only
        sim.time_loop(1)
        assert rt.used() < before
        assert stage_kernels(rt)["k_stage_split"] == 3


# ------------------------------------------------------------------ the network's two copies
def test_inference_uses_the_parameters_on_the_device(rt):
    """A training call that changes the parameters and then fails: the FP32 layers that later launches
    take by value are those of the device, in the batch, the inference and the step."""
    cfg, h = problem("mhd")
    cfg = cfg.replace(precision="fp32_split", eos_guess="mlp_rescue")
    rt.watch("k_mlp_train_step", "PPPPPPiPP")
    # first word of the by-value layers: W1[0]
    rt.watch("k_eos_guess", "si")
    rt.watch("k_mlp_infer", "i")
    rt.watch("k_c2p_rescue", "si")
    bits = lambda x: int(np.float32(x).view(np.int32))
    last = lambda k: rt.launches_of(k)[-1][1][1 if k != "k_mlp_infer" else 0]
    from phlegethon_b200.abi import Simulation
    with Simulation(cfg, tiny_table(cfg)) as sim:
        sim.upload(h)
        sim.init_thermo()
        sim.compute_hyperbolic_dt()
        w = np.zeros(4545, np.float32)
        w[0] = 1.0
        assert sim.lib.phl_mlp_set_params(sim.ctx, w.ctypes.data_as(C.POINTER(C.c_float))) == 0
        sim.time_loop(1)
        assert last("k_c2p_rescue") == bits(1.0)
        n = 16
        a = [np.ones(n) for _ in range(7)]
        feat, out = np.zeros((n, 4), np.float32), np.zeros(n, np.float32)
        calls = (("k_eos_guess", lambda: sim.lib.phl_eos_invert_batch(sim.ctx, n, *[x.ctypes.data for x in a], None, 1)),
                 ("k_mlp_infer", lambda: sim.lib.phl_mlp_infer_device(sim.ctx, n, feat.ctypes.data, out.ctypes.data)),
                 ("k_c2p_rescue", lambda: sim.lib.phl_run_steps(sim.ctx, 1, np.inf, None, None)),
                 ("k_c2p_rescue", lambda: sim.lib.phl_hydro_step(sim.ctx)))
        for q, (kernel, call) in enumerate(calls):
            rt.refuse_downloads(1000)
            assert sim.lib.phl_mlp_train(sim.ctx, 256, 1, 1, 64, 1e-3, None) == -2
            params = rt.launches_of("k_mlp_train_step")[-1][1][0]
            C.c_float.from_address(params).value = 2.0 + q  # what the updates would have done
            assert call() == -2  # not with layers of two networks
            rt.refuse_downloads(0)
            assert call() == 0
            assert last(kernel) == bits(2.0 + q), kernel


# ------------------------------------------------------------------ graphs of the driver's steps
def test_hydro_step_graphs_are_made_once(rt):
    """A graph a buffer parity after eight calls; none for a driver that uploads its whole state, background
    included, before every step."""
    cfg, h = problem("bubble")
    with started(cfg, h) as sim:
        for _ in range(30):
            sim.hydro_step()
        assert rt.instantiations() == 2  # three stages: the parity alternates
        for _ in range(30):
            sim.upload(h)
            sim.hydro_step()
        assert rt.instantiations() == 2


def test_hydro_step_without_room_for_a_graph(rt):
    """A driver that has given all device memory to a pool of its own: hydro_step goes on launching."""
    cfg, h = problem("bubble")
    rt.watch("k_c2p", "s")
    with started(cfg, h) as sim:
        rt.refuse_graphs(1000)
        for _ in range(30):
            sim.hydro_step()
        # three stages a call; a try that failed has captured its launches as well
        assert rt.instantiations() == 0 and len(rt.launches_of("k_c2p")) >= 3 * 30
        rt.refuse_graphs(0)
        for _ in range(12):
            sim.hydro_step()
        assert rt.instantiations() > 0
