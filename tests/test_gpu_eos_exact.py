"""Bit-exactness of the FP64 Helmholtz evaluations where they take short cuts: the table cell found
without a logarithm (states on, next to and between the table's nodes), quotients by
multiplication with a known reciprocal, and energies at temperature nodes (bracket guess)."""
import ctypes as C
from fractions import Fraction

import numpy as np
import pytest

from phlegethon_b200 import helm_table, problems


def test_division_by_known_reciprocal_rounds_correctly():
    """Two quotient corrections with exact residuals from RN(1/b) give RN(a/b): the five operations of
    the device function, each rounded exactly (Fraction to float rounds to nearest even)."""
    rng = np.random.default_rng(3)
    n = 20000
    a = rng.uniform(1, 2, n) * 10.0 ** rng.uniform(-60, 60, n) * rng.choice([-1.0, 1.0], n)
    b = rng.uniform(1, 2, n) * 10.0 ** rng.uniform(-25, 55, n)
    # significands next to a power of two, where a quotient is hardest to round
    b[::5] = np.nextafter(2.0 ** rng.integers(-60, 60, b[::5].size), rng.choice([0.0, np.inf], b[::5].size))
    fma = lambda x, y, z: float(Fraction(x) * Fraction(y) + Fraction(z))
    for x, y in zip(a.tolist(), b.tolist()):
        r = 1.0 / y
        q = x * r
        q = fma(fma(-y, q, x), r, q)
        q = fma(fma(-y, q, x), r, q)
        assert q == x / y, (x.hex(), y.hex())


def _states():
    """(rho, T, abar, zbar) on the nodes, an ulp and about 1e-12 next to them, and in between."""
    rho, T, _, _ = helm_table.nodes(**helm_table.X1_TABLE)
    rng = np.random.default_rng(5)

    def near(x, n):
        v = x[rng.integers(1, x.size - 1, n)]
        k = rng.integers(0, 8, n)
        out = v.copy()
        out = np.where(k == 1, np.nextafter(v, np.inf), out)
        out = np.where(k == 2, np.nextafter(v, 0.0), out)
        out = np.where(k == 3, v * (1 + 1e-12), out)
        out = np.where(k == 4, v * (1 - 1e-12), out)
        out = np.where(k == 5, v * (1 + 3e-12), out)
        out = np.where(k == 6, v * (1 - 3e-12), out)
        return np.where(k == 7, v * 10.0 ** rng.uniform(0, 0.1, n), out)
    n = 3000
    zbar = np.where(rng.random(n) < 0.5, 1.0, rng.uniform(1, 28, n))
    abar = np.where(rng.random(n) < 0.5, zbar, 2.1 * zbar)
    d, t = near(rho[40:240], n), near(T[10:80], n)
    return d * abar / zbar, t, abar, zbar


@pytest.mark.gpu
def test_energy_bitwise_at_and_around_the_nodes(gpu_lib):
    import pyoracle
    import torch
    from phlegethon_b200.abi import Simulation
    tab = helm_table.generate(**helm_table.X1_TABLE)
    cfg, _ = problems.stratified_3d(8, table=helm_table.X1_TABLE)
    helm = pyoracle.Helm.for_config(cfg, *tab)
    s = _states()
    want = np.array([helm.given2(*q, deriv=False)[0] for q in zip(*s)])
    with Simulation(cfg, tab) as sim:
        d = [torch.from_numpy(np.ascontiguousarray(v)).cuda() for v in s]
        e = torch.zeros(len(want), dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        assert sim.lib.phl_eos_energy_device(sim.ctx, len(want), d[0].data_ptr(), d[1].data_ptr(), d[2].data_ptr(),
                                             d[3].data_ptr(), e.data_ptr()) == 0
        got = e.cpu().numpy()
    # the oracle's log10 and the device's may put a state within a few ulp of a node into either cell,
    # whose interpolants meet there to rounding; everywhere else the bits agree.  The logarithms, the step
    # and the nodes' own powers are off by a few ulp of log10 x, which is x to some 1e-14
    rho_n, T_n, _, _ = helm_table.nodes(**helm_table.X1_TABLE)
    dist = lambda x, nodes: np.abs(x[:, None] / nodes[None, :] - 1.0).min(axis=1)
    on_node = np.minimum(dist(s[0] * (s[3] / s[2]), rho_n), dist(s[1], T_n)) < 2e-13
    same = got.view(np.int64) == want.view(np.int64)
    assert np.all(same[~on_node])
    assert np.all(np.abs(got - want) <= 1e-13 * np.abs(want))
    # states of both kinds: five of eight draws of T, and of rho Ye, stay off their node by 1e-12 and more
    assert on_node.mean() > 0.5 and (~on_node).mean() > 0.3


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 127, 129, 1000])
def test_bracket_inversion_bitwise(gpu_lib, n):
    """The bracket guess and the Newton against the oracle bit for bit, block remainders included."""
    import pyoracle
    from phlegethon_b200.abi import Simulation
    tab = helm_table.generate(**helm_table.X1_TABLE)
    cfg, _ = problems.stratified_3d(8, table=helm_table.X1_TABLE)
    helm = pyoracle.Helm.for_config(cfg, *tab)
    rho, T, abar, zbar = problems.eos_samples(n, seed=n)
    e = np.array([helm.given2(*q, deriv=False)[0] for q in zip(rho, T, abar, zbar)])
    out, it = np.zeros(n), np.zeros(n, dtype=np.int32)
    with Simulation(cfg, tab) as sim:
        rc = sim.lib.phl_eos_invert_batch(sim.ctx, n, *[a.ctypes.data for a in (rho, e, abar, zbar)], out.ctypes.data,
                                          None, None, it.ctypes.data, 2)
        assert rc == 0
    T_want, it_want = helm.invert_batch(rho, e, abar, zbar, guess=2)
    assert np.array_equal(out, T_want) and np.array_equal(it, it_want)


@pytest.mark.gpu
@pytest.mark.parametrize("out", [False, True])
@pytest.mark.parametrize("n,off", [(1, 0.0), (129, 1e-3), (1000, 0.3), (1000, 0.0)])
def test_warm_inversion_bitwise(gpu_lib, n, off, out):
    """The Newton from a warm start against the oracle bit for bit, with p and cs and without (the two are
    kernels of their own); p and cs are those of the bracket guess where T is the same."""
    import pyoracle
    from phlegethon_b200.abi import Simulation
    tab = helm_table.generate(**helm_table.X1_TABLE)
    cfg, _ = problems.stratified_3d(8, table=helm_table.X1_TABLE)
    helm = pyoracle.Helm.for_config(cfg, *tab)
    rho, T, abar, zbar = problems.eos_samples(n, seed=n + 1)
    e = np.array([helm.given2(*q, deriv=False)[0] for q in zip(rho, T, abar, zbar)])
    T0 = T * (1.0 + off)
    got, it, p, cs = T0.copy(), np.zeros(n, dtype=np.int32), np.zeros(n), np.zeros(n)
    with Simulation(cfg, tab) as sim:
        def invert(t, pp, cc, guess):
            po = (pp.ctypes.data, cc.ctypes.data) if pp is not None else (None, None)
            assert sim.lib.phl_eos_invert_batch(sim.ctx, n, *[a.ctypes.data for a in (rho, e, abar, zbar)], t.ctypes.data,
                                                *po, it.ctypes.data, guess) == 0
        tb, pb, cb = np.zeros(n), np.zeros(n), np.zeros(n)
        invert(tb, pb, cb, 2)
        invert(got, p if out else None, cs if out else None, 0)
    T_want, it_want = helm.invert_batch(rho, e, abar, zbar, T0=T0, guess=0)
    assert np.array_equal(got, T_want) and np.array_equal(it, it_want)
    if out:
        same = got == tb
        assert np.all(p > 0.0) and np.all(cs > 0.0)
        assert np.array_equal(p[same], pb[same]) and np.array_equal(cs[same], cb[same])
