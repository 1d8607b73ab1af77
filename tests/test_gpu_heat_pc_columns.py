"""Piecewise-constant float32 heat at the edges of its column groups: widths that
end inside, at and after a group of four, one-row and one-plane grids, both
block shapes, every coordinate system.  Residual against the oracle (rel L-inf
2e-6, the float32 bound of the residual tests)."""
import numpy as np
import pytest

from oracle import fvm_oracle as O
from tests.helpers import rel_linf, to_fp32

pytestmark = pytest.mark.gpu

PRM = {"mass_density": 2.0, "specific_heat_capacity": 3.0, "thermal_conductivity": 0.7, "volumetric_heat_source": 0.25}


@pytest.mark.parametrize("coords", ["cartesian", "cylindrical", "spherical"])
@pytest.mark.parametrize("tile_ty", [0, 8])
@pytest.mark.parametrize("n", [(1, 1, 1), (2, 5, 3), (3, 17, 2), (4, 8, 9), (29, 9, 4), (33, 16, 5), (35, 7, 6), (66, 19, 7)],
                         ids=lambda n: "x".join(map(str, n)))
def test_residual(n, tile_ty, coords):
    from multiphysics_fvm_b200.backend import SIDES, Simulation
    from multiphysics_fvm_b200.grid import boundary_conditions as bc
    from multiphysics_fvm_b200.numerics import reconstructors, time_integrators
    cfg = {"x1_min": 0.5, "x1_max": 1.5, "x2_min": 0.6, "x2_max": 2.2, "x3_min": 0.0, "x3_max": 1.0,
           "nx1": n[0], "nx2": n[1], "nx3": n[2]}
    sim = Simulation("heat", coords, cfg, PRM, {"reconstructor": reconstructors.piecewise_constant},
                     {"internal_energy_density": {s: bc.neumann for s in SIDES}}, time_integrators.rk3_ssp,
                     precision="fp32", tile_ty=tile_ty)
    U = to_fp32(np.random.default_rng(8).uniform(6.0, 12.0, (1,) + tuple(x + 2 for x in n)))
    sim.upload(U)
    ref = O.heat_rhs(U, O.Geometry(coords, cfg), PRM, dict(reconstructor="piecewise_constant", slope_limiter=None))
    assert rel_linf(sim.residual(), ref) <= 2e-6
