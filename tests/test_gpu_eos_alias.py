"""The batch inversion with its temperature array also an input array: every sample is read before its
result is written, whatever the guess."""
import numpy as np
import pytest

from phlegethon_b200 import helm_table, problems

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("guess", [1, 2])
@pytest.mark.parametrize("n", [1, 130, 4097])
def test_output_may_alias_an_input(gpu_lib, table, guess, n):
    import torch
    from phlegethon_b200.abi import Simulation
    cfg, _ = problems.stratified_3d(8)
    rho, T, abar, zbar = problems.eos_samples(n, seed=3)
    with Simulation(cfg, table) as sim:
        assert sim.lib.phl_mlp_train(sim.ctx, 1 << 16, 5, 1, 8192, 1e-3, None) == 0
        d = [torch.from_numpy(np.ascontiguousarray(v)).cuda() for v in (rho, T, abar, zbar)]
        e = torch.zeros(n, dtype=torch.float64, device="cuda")
        out = torch.zeros(n, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        assert sim.lib.phl_eos_energy_device(sim.ctx, n, d[0].data_ptr(), d[1].data_ptr(), d[2].data_ptr(),
                                             d[3].data_ptr(), e.data_ptr()) == 0

        def invert(to):
            rc = sim.lib.phl_eos_invert_batch_device(sim.ctx, n, d[0].data_ptr(), e.data_ptr(), d[2].data_ptr(),
                                                     d[3].data_ptr(), to.data_ptr(), None, None, None, guess)
            assert rc == 0
        invert(out)
        invert(e)
        assert torch.equal(out, e)
