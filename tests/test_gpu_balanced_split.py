"""The balanced split of a stage's work (depth 0) against fixed z-march depths:
every cell's arithmetic is the same whatever block and piece it falls into, so
the states agree bitwise.  Sizes: one unit of work, fewer units than resident
blocks, runs that cross column boundaries, partial edge tiles, one-plane grids."""
import math

import numpy as np
import pytest

from helpers import random_ns_state, to_fp32

pytestmark = pytest.mark.gpu

SIZES = [(5, 4, 1), (33, 9, 2), (31, 70, 67), (97, 33, 40), (64, 300, 1), (40, 24, 200)]
FAMILIES = [("navier_stokes", "cartesian", "fp32", "van_leer", 0.0), ("navier_stokes", "cartesian", "fp32", "minmod", 1e-3),
            ("navier_stokes", "cylindrical", "fp32", "van_leer", 1e-3), ("navier_stokes", "spherical", "fp64", "minmod", 0.0),
            ("navier_stokes", "cartesian", "fp64", "van_leer", 1e-3),
            ("heat", "cylindrical", "fp32", None, 0.0), ("heat", "cartesian", "fp32", "minmod", 0.0),
            ("heat", "spherical", "fp64", None, 0.0), ("maxwell", "spherical", "fp32", "monotonized_central", 0.0),
            ("maxwell", "cartesian", "fp64", "minmod", 0.0)]


def _sim(family, n, zchunk):
    from multiphysics_fvm_b200.backend import SIDES, VARIABLES, Simulation
    from multiphysics_fvm_b200.grid import boundary_conditions as bc
    from multiphysics_fvm_b200.numerics import reconstructors, riemann_solvers, slope_limiters, time_integrators
    physics, coords, precision, lim, mu = family
    prm = {"navier_stokes": {"heat_capacity_ratio": 1.4, "dynamic_viscosity": mu,
                             "gravitational_acceleration": [0.0, 0.1, -0.2]},
           "heat": {"mass_density": 1.0, "specific_heat_capacity": 1.0, "thermal_conductivity": 1.0,
                    "volumetric_heat_source": 0.1},
           "maxwell": {"magnetic_permeability": 1.0, "electric_permittivity": 1.0, "electrical_conductivity": 0.1,
                       "charge_density": 0.0, "magnetic_cleaning_coeff": 0.01, "electric_cleaning_coeff": 0.01}}[physics]
    cfg = {"x1_min": 0.5, "x1_max": 1.5, "x2_min": 0.6, "x2_max": 2.2, "x3_min": 0.0, "x3_max": 1.0,
           "nx1": n[0], "nx2": n[1], "nx3": n[2]}
    schemes = {"riemann_solver": riemann_solvers.hll,
               "reconstructor": reconstructors.muscl if lim else reconstructors.piecewise_constant,
               "slope_limiter": getattr(slope_limiters, lim or "minmod")}
    bcs = {v: {s: (bc.neumann if s in ("left", "right") else bc.periodic) for s in SIDES} for v in VARIABLES[physics]}
    return Simulation(physics, coords, cfg, prm, schemes, bcs, time_integrators.rk3, precision=precision, zchunk=zchunk)


@pytest.mark.parametrize("n", SIZES, ids=lambda n: "x".join(map(str, n)))
@pytest.mark.parametrize("family", FAMILIES, ids=lambda f: "-".join(map(str, f)))
def test_balanced_equals_fixed_depth(family, n):
    rng = np.random.default_rng(3)
    shape = tuple(x + 2 for x in n)
    if family[0] == "navier_stokes":
        U = random_ns_state(shape, rng)
    else:
        U = rng.uniform(1.0, 2.0, ((1 if family[0] == "heat" else 6),) + shape)
    U = to_fp32(U)
    outs = []
    for z in (0, 3, max(n[2], 1)):
        sim = _sim(family, n, z)
        sim.upload(U)
        sim.set_time(0.0, math.inf, 0.2)
        sim.step(2)
        assert sim.status() == 0
        outs.append(sim.download())
        sim.close()
    assert np.array_equal(outs[0], outs[1]) and np.array_equal(outs[0], outs[2])
