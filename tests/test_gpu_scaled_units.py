"""States in units far from one.  Scaling mass, length and time by powers of two
changes only float32 exponents, so a float32 residual is that of the unit state
times a power of two, up to the rounding of a different exponent's reciprocal
and square root (relative L-inf <= 1e-6 allowed).

* thin: densities of 2^-104 (5e-32) with velocities of 2^47, energies of 2^-10;
* strong: nearly uniform states of 2^36 (momentum) and 2^72 (energy), 2^72 for
  fields: the differences between cells are in range, the product of a ghost
  cell's two differences, whose slope is not used, is above float32's largest."""
import numpy as np
import pytest

from tests.helpers import bcs_dict, random_ns_state, rel_linf, to_fp32

pytestmark = pytest.mark.gpu


def _residual(physics, n, coords, limiter, riemann, prm, U):
    from multiphysics_fvm_b200.backend import Simulation
    from multiphysics_fvm_b200.numerics import reconstructors, riemann_solvers, slope_limiters, time_integrators
    cfg = dict(x1_min=1.0, x1_max=2.0, x2_min=0.6, x2_max=1.4, x3_min=0.0, x3_max=0.6, nx1=n[0], nx2=n[1], nx3=n[2])
    sim = Simulation(physics, coords, cfg, prm,
                     {"reconstructor": reconstructors.muscl, "slope_limiter": getattr(slope_limiters, limiter),
                      "riemann_solver": getattr(riemann_solvers, riemann)},
                     bcs_dict(physics, [["periodic"] * 6] * U.shape[0]), time_integrators.rk3, precision="fp32")
    sim.upload(U)
    r = sim.residual()
    assert sim.status() == 0
    sim.close()
    return r


def _ns(mu):
    return {"heat_capacity_ratio": 1.4, "dynamic_viscosity": mu, "gravitational_acceleration": [0.0, 0.0, 0.0]}


@pytest.mark.parametrize("n", [(40, 20, 12), (70, 33, 1)], ids=str)
@pytest.mark.parametrize("mu", [0.0, 2.0 ** -10], ids=["inviscid", "viscous"])
@pytest.mark.parametrize("a,b,smooth,limiter,riemann",
                         [(-104, 47, False, "minmod", "hll"), (-104, 47, False, "monotonized_central", "rusanov"),
                          (0, 36, True, "van_leer", "hll"), (0, 36, True, "van_leer", "rusanov"),
                          (0, 36, True, "minmod", "hll"), (0, 36, True, "monotonized_central", "hll")],
                         ids=["thin-minmod", "thin-mc", "strong-van_leer", "strong-van_leer-rusanov",
                              "strong-minmod", "strong-mc"])
def test_navier_stokes(a, b, smooth, limiter, riemann, mu, n):
    """Density times 2^a, velocity times 2^b."""
    U = random_ns_state(tuple(x + 2 for x in n), np.random.default_rng(5))
    if smooth:
        U = U.mean((1, 2, 3), keepdims=True) * (1 + 1e-4 * (U - U.mean((1, 2, 3), keepdims=True)))
    U = to_fp32(U)
    scale = np.array([a, a + b, a + b, a + b, a + 2 * b], dtype=np.float64).reshape(5, 1, 1, 1)
    ref = _residual("navier_stokes", n, "cartesian", limiter, riemann, _ns(mu), U)
    got = _residual("navier_stokes", n, "cartesian", limiter, riemann, _ns(mu * 2.0 ** (a + b)), U * 2.0 ** scale)
    got = got * 2.0 ** -(scale + b)
    assert np.all(np.isfinite(got))
    for q in range(5):
        assert rel_linf(got[q], ref[q]) <= 1e-6


@pytest.mark.parametrize("limiter", ["van_leer", "minmod", "monotonized_central"])
def test_maxwell(limiter):
    n = (40, 20, 12)
    prm = {"magnetic_permeability": 1.0, "electric_permittivity": 1.0, "electrical_conductivity": 0.0,
           "charge_density": 0.0, "magnetic_cleaning_coeff": 0.001, "electric_cleaning_coeff": 0.001}
    U = to_fp32(1 + 1e-4 * np.random.default_rng(5).uniform(-1, 1, (6,) + tuple(x + 2 for x in n)))
    ref = _residual("maxwell", n, "cartesian", limiter, "rusanov", prm, U)
    got = _residual("maxwell", n, "cartesian", limiter, "rusanov", prm, U * 2.0 ** 72) * 2.0 ** -72
    assert np.all(np.isfinite(got)) and rel_linf(got, ref) <= 1e-6
