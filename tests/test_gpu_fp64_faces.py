"""The FP64 form's face kernels at the edges of their splits, bit for bit against the oracle: warp rows
of 29 faces along x1 (row lengths around multiples of 29, walls along x1), and the walks that grids
of a million cells take."""
import numpy as np
import pytest

from phlegethon_b200 import problems
from util import max_abs_diff, permute_axes

pytestmark = pytest.mark.gpu


def run_both(cfg, h, table, steps):
    import pyoracle
    from phlegethon_b200.abi import Simulation
    hg, ho = h.copy(), h.copy()
    with Simulation(cfg, table if cfg.helmholtz else None) as sim:
        sim.upload(hg)
        sim.init_thermo()
        sim.compute_hyperbolic_dt()
        sim.time_loop(steps)
        sim.download(hg)
    helm = pyoracle.Helm.for_config(cfg, *table) if cfg.helmholtz else None
    o = pyoracle.OracleGrid(ho, helm) if helm else pyoracle.OracleGrid(ho)
    o.init_thermo()
    o.compute_hyperbolic_dt()
    o.time_loop(steps)
    return hg, ho


@pytest.mark.parametrize("n", [4, 27, 28, 29, 57, 58])
@pytest.mark.parametrize("mhd", [False, True])
def test_rows(gpu_lib, oracle, table, n, mhd):
    cfg, h = problems.stratified_3d(n, ny=6, nz=5, mhd=mhd, seed=n)
    assert max_abs_diff(*run_both(cfg, h, table, 2)) == 0.0


@pytest.mark.parametrize("perm", [(1, 0, 2), (0, 2, 1)])
def test_walls_along_x1_and_x3(gpu_lib, oracle, table, perm):
    cfg, h = problems.stratified_3d(9, ny=31, nz=6, mhd=True)
    h = permute_axes(h, perm)
    assert max_abs_diff(*run_both(h.cfg, h, table, 2)) == 0.0


@pytest.mark.parametrize("n", [29, 59])
def test_rows_2d(gpu_lib, oracle, n):
    cfg, h = problems.hot_bubble_2d(n)
    assert max_abs_diff(*run_both(cfg, h, None, 4)) == 0.0
    cfg, h = problems.orszag_tang_2d(n)
    assert max_abs_diff(*run_both(cfg, h, None, 4)) == 0.0


def test_walks_of_large_grids(gpu_lib, oracle, table):
    """1,006,740 cells, x2 and x3 extents on and off multiples of 8."""
    cfg, h = problems.stratified_3d(105, ny=102, nz=94, mhd=True)
    assert cfg.n_cells >= 1000000
    assert max_abs_diff(*run_both(cfg, h, table, 1)) == 0.0
