"""Host transfers through the pinned chunks: states smaller than a chunk, of a few
chunks and of several threads' worth, as one array and as the reference's dict,
pageable and page-locked.  Every way gives the same bytes: the interior as
uploaded, ghost faces, edges and corners as the oracle fills them."""
import numpy as np
import pytest

from oracle import fvm_oracle as O
from tests.helpers import bcs_dict, oracle_bcs

pytestmark = pytest.mark.gpu

KINDS = [["periodic"] * 2 + ["neumann", ("dirichlet", 1.5)] + ["reflecting", "neumann"]] * 5
I3 = (slice(None),) + (slice(1, -1),) * 3


@pytest.mark.parametrize("n", [(1, 1, 1), (3, 2, 4), (31, 40, 29), (64, 63, 61), (97, 100, 128)],
                         ids=lambda n: "x".join(map(str, n)))
def test_every_way_gives_the_same_bytes(n):
    import torch
    from multiphysics_fvm_b200.backend import Simulation
    from multiphysics_fvm_b200.numerics import reconstructors, riemann_solvers, slope_limiters, time_integrators
    cfg = dict(x1_min=0.0, x1_max=1.0, x2_min=0.0, x2_max=0.8, x3_min=0.0, x3_max=0.6, nx1=n[0], nx2=n[1], nx3=n[2])
    sim = Simulation("navier_stokes", "cartesian", cfg,
                     {"heat_capacity_ratio": 1.4, "dynamic_viscosity": 0.0, "gravitational_acceleration": [0.0] * 3},
                     {"reconstructor": reconstructors.muscl, "slope_limiter": slope_limiters.minmod,
                      "riemann_solver": riemann_solvers.hll}, bcs_dict("navier_stokes", KINDS),
                     time_integrators.rk3_ssp, precision="fp64")
    rng = np.random.default_rng(1)
    shape = (5,) + tuple(x + 2 for x in n)
    for way in ("array", "dict", "pinned", "strided"):
        U = rng.uniform(1.0, 2.0, shape)
        ref = U.copy()
        O.apply_bcs(ref, oracle_bcs(KINDS))
        if way == "array":
            sim.upload(U)
        elif way == "dict":
            sim.upload(dict(zip(sim.variables, U)))
        elif way == "pinned":
            sim.upload(torch.from_numpy(U).pin_memory().numpy())
        else:
            sim.upload({k: np.asfortranarray(v) for k, v in zip(sim.variables, U)})
        got = sim.download()
        assert np.array_equal(got, ref)
        D = {k: np.empty(shape[1:]) for k in sim.variables}
        sim.download_into(D)
        F = {k: np.empty(shape[1:], order="F") for k in sim.variables}
        sim.download_into(F)
        P = torch.empty(shape, dtype=torch.float64).pin_memory().numpy()
        sim.download(P)
        for q, k in enumerate(sim.variables):
            assert np.array_equal(D[k], ref[q]) and np.array_equal(F[k], ref[q])
        assert np.array_equal(P, ref)
    with pytest.raises(ValueError):
        sim.upload({k: np.zeros((2, 2, 2)) for k in sim.variables})
