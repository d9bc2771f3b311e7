"""The assembled matrix read back to device and to host memory."""
import numpy as np
import pytest

from conftest import to_dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nb", [1, 255, 256, 257, 1000])
def test_blocks_out_to_device_and_host(solver, cuda, nb):
    import torch

    rng = np.random.default_rng(nb)
    idx = np.arange(nb, dtype=np.int32)
    vals = rng.normal(size=(nb, 9))
    solver.assemble(nb, to_dev(idx, cuda), to_dev(idx, cuda), to_dev(vals, cuda))
    d = torch.full((nb + 1, 9), 7.0, dtype=torch.float64, device=cuda)
    solver._check(solver.lib.b2s_get_upper_bsr(solver.h, None, None, d.data_ptr()))
    assert np.array_equal(d[:nb].cpu().numpy(), vals) and (d[nb] == 7.0).all()
    assert np.array_equal(solver.upper_bsr()[2], vals)
