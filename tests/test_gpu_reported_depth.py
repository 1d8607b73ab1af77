"""The z-march depth that a handle reports (fvm_tiling, fvm_autotune) is one to
ask for: a handle made with it runs its steps in about the time of the handle
that reported it.  1.2 times is allowed; the longest run of the default split,
asked for as a fixed depth, leaves a second round of blocks: 1.25 to 1.29 times
on the first two grids."""
import math

import numpy as np
import pytest

from tests.helpers import bcs_dict, random_ns_state

pytestmark = pytest.mark.gpu


def _sim(n, precision, zchunk=0):
    from multiphysics_fvm_b200.backend import Simulation
    from multiphysics_fvm_b200.numerics import reconstructors, riemann_solvers, slope_limiters, time_integrators
    cfg = dict(x1_min=0, x1_max=1, x2_min=0, x2_max=1, x3_min=0, x3_max=1, nx1=n[0], nx2=n[1], nx3=n[2])
    sim = Simulation("navier_stokes", "cartesian", cfg,
                     {"heat_capacity_ratio": 1.4, "dynamic_viscosity": 0.0, "gravitational_acceleration": [0, 0, 0]},
                     {"reconstructor": reconstructors.muscl, "slope_limiter": slope_limiters.minmod,
                      "riemann_solver": riemann_solvers.hll},
                     bcs_dict("navier_stokes", [["periodic"] * 6] * 5), time_integrators.rk3_ssp,
                     precision=precision, zchunk=zchunk)
    sim.upload(random_ns_state(tuple(x + 2 for x in n), np.random.default_rng(1)))
    sim.set_time(0.0, math.inf, 0.01)
    return sim


def _stage_ms(sim):
    sim.step(2)
    return min(sim.profile_steps(3)[0] for _ in range(5))


@pytest.mark.parametrize("tuned", [False, True])
@pytest.mark.parametrize("n,precision", [((128, 128, 128), "fp32"), ((256, 256, 256), "fp32"), ((97, 130, 61), "fp32"),
                                         ((96, 96, 96), "fp64")])
def test_asking_for_the_reported_depth(n, precision, tuned):
    sim = _sim(n, precision)
    z = sim.autotune()[0] if tuned else sim.tiling()[1]
    assert sim.tiling()[1] == z and 1 <= z <= n[2]
    rows, t = sim.tiling()[0], _stage_ms(sim)
    sim.close()
    fixed = _sim(n, precision, zchunk=z)
    assert fixed.tiling()[1] == z
    if fixed.tiling()[0] == rows:
        assert _stage_ms(fixed) <= 1.2 * t
    fixed.close()
