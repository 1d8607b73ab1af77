"""Dense state copies at the edges of their vector width: rows that are and are
not whole 16-byte groups, rows shorter and longer than a warp's reach, and a
dense tensor whose base is not 16-byte aligned.  A copy up and back is exact."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("n", [(4, 1, 1), (5, 3, 2), (12, 7, 33), (128, 5, 9), (132, 40, 3), (131, 4, 6)])
def test_round_trip(n, offset):
    import torch
    from multiphysics_fvm_b200 import closure as CL
    from multiphysics_fvm_b200.backend import Simulation
    from multiphysics_fvm_b200.setups import kelvin_helmholtz_sharp as kh
    sim = Simulation.from_setup(kh.get_setup(*n, precision="fp32"))
    shape = (5, n[2], n[1], n[0])
    size = int(np.prod(shape))
    src = torch.empty(size + offset, device="cuda")[offset:].view(shape)
    src.copy_(torch.rand(shape, device="cuda"))
    out = torch.zeros(size + offset, device="cuda")[offset:].view(shape)
    CL.upload_dense(sim, src)
    CL.download_dense(sim, out)
    assert torch.equal(src, out)
    host = sim.download()[:, 1:-1, 1:-1, 1:-1]
    assert np.array_equal(host, src.permute(0, 3, 2, 1).cpu().numpy().astype(np.float64))
