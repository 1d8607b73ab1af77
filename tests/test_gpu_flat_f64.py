"""Float64 one-plane grids, whose steps leave out the x3 pipeline: two steps
against the oracle, which runs it, for both x3 boundaries that copy the plane
and one that does not."""
import numpy as np
import pytest

from oracle import fvm_oracle as O
from tests.helpers import bcs_dict, oracle_bcs, random_ns_state, rel_linf

pytestmark = pytest.mark.gpu

PRM = {"heat_capacity_ratio": 1.4, "dynamic_viscosity": 0.0, "gravitational_acceleration": [0.1, -0.2, 0.3]}


@pytest.mark.parametrize("limiter,riemann", [("minmod", "hll"), ("monotonized_central", "rusanov"), ("van_leer", "hll")])
@pytest.mark.parametrize("x3", ["periodic", "neumann", "reflecting"])
@pytest.mark.parametrize("n", [(5, 4), (33, 9), (70, 31)])
def test_against_oracle(n, x3, limiter, riemann):
    from multiphysics_fvm_b200.backend import Simulation
    from multiphysics_fvm_b200.numerics import reconstructors, riemann_solvers, slope_limiters, time_integrators
    cfg = dict(x1_min=0.0, x1_max=1.0, x2_min=0.0, x2_max=0.8, x3_min=0.0, x3_max=0.6, nx1=n[0], nx2=n[1], nx3=1)
    kinds = [["periodic"] * 2 + ["neumann"] * 2 + [x3] * 2] * 5
    U = random_ns_state((n[0] + 2, n[1] + 2, 3), np.random.default_rng(4))
    sim = Simulation("navier_stokes", "cartesian", cfg, PRM,
                     {"reconstructor": reconstructors.muscl, "slope_limiter": getattr(slope_limiters, limiter),
                      "riemann_solver": getattr(riemann_solvers, riemann)},
                     bcs_dict("navier_stokes", kinds), time_integrators.rk3_ssp, precision="fp64")
    sim.upload(U)
    sim.step(2, dt=1e-3)
    assert sim.status() == 0
    O.run("navier_stokes", U, PRM, O.Geometry("cartesian", cfg),
          dict(reconstructor="muscl", slope_limiter=limiter, riemann_solver=riemann), oracle_bcs(kinds), "rk3_ssp", 0.4,
          2, dt_fixed=1e-3)
    I3 = (slice(None),) + (slice(1, -1),) * 3
    assert rel_linf(sim.download()[I3], U[I3]) <= 1e-12
