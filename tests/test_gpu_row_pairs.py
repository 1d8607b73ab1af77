"""Float32 inviscid grids whose row count leaves the last strip of two rows half
filled, or is below one strip, with one-plane grids (their own march) and every
coordinate system: two steps against the float64 oracle from the same float32
state, relative L-inf <= 1e-5 (a few float32 roundings of the state a stage)."""
import numpy as np
import pytest

from oracle import fvm_oracle as O
from tests.helpers import bcs_dict, oracle_bcs, random_ns_state, rel_linf, to_fp32

pytestmark = pytest.mark.gpu

PRM = {"heat_capacity_ratio": 1.4, "dynamic_viscosity": 0.0, "gravitational_acceleration": [0.1, -0.2, 0.3]}


@pytest.mark.parametrize("coords", ["cartesian", "cylindrical", "spherical"])
@pytest.mark.parametrize("n", [(1, 1, 1), (33, 1, 4), (31, 2, 1), (32, 7, 3), (65, 9, 1), (5, 17, 2)])
def test_against_oracle(n, coords):
    from multiphysics_fvm_b200.backend import Simulation
    from multiphysics_fvm_b200.numerics import reconstructors, riemann_solvers, slope_limiters, time_integrators
    cfg = dict(x1_min=1.0, x1_max=2.0, x2_min=0.6, x2_max=1.4, x3_min=0.0, x3_max=0.6, nx1=n[0], nx2=n[1], nx3=n[2])
    kinds = [["neumann"] * 4 + ["periodic"] * 2] * 5
    U = to_fp32(random_ns_state(tuple(k + 2 for k in n), np.random.default_rng(11)))
    sim = Simulation("navier_stokes", coords, cfg, PRM,
                     {"reconstructor": reconstructors.muscl, "slope_limiter": slope_limiters.van_leer,
                      "riemann_solver": riemann_solvers.hll},
                     bcs_dict("navier_stokes", kinds), time_integrators.rk4, precision="fp32")
    sim.upload(U)
    sim.step(2, dt=1e-4)
    assert sim.status() == 0
    O.run("navier_stokes", U, PRM, O.Geometry(coords, cfg),
          dict(reconstructor="muscl", slope_limiter="van_leer", riemann_solver="hll"), oracle_bcs(kinds), "rk4", 0.4, 2,
          dt_fixed=1e-4)
    I3 = (slice(None),) + (slice(1, -1),) * 3
    assert rel_linf(sim.download()[I3], U[I3]) <= 1e-5
