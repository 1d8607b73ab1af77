"""Float32 Navier-Stokes rounding, held to what it was before the kernels were
rearranged for speed: relative L2 error of a state after some steps of smooth flow
against the float64 oracle from the same float32 state.  The runs are
deterministic; the bounds are the errors of before."""
import numpy as np
import pytest

from oracle import fvm_oracle as O
from tests.helpers import bcs_dict, oracle_bcs, to_fp32

pytestmark = pytest.mark.gpu


def error(coords, n, lo, hi, mu, limiter, steps, dt):
    from multiphysics_fvm_b200.backend import Simulation
    from multiphysics_fvm_b200.numerics import reconstructors, riemann_solvers, slope_limiters, time_integrators
    cfg = {f"x{a + 1}_{m}": v[a] for a in range(3) for m, v in (("min", lo), ("max", hi))}
    cfg |= {f"nx{a + 1}": n[a] for a in range(3)}
    x = [2 * np.pi * (np.arange(k + 2) - 0.5) / k for k in n]
    x, y, z = x[0][:, None, None], x[1][None, :, None], x[2][None, None, :]
    rng = np.random.default_rng(8)
    noise = lambda: 1e-3 * rng.uniform(-1, 1, tuple(k + 2 for k in n))  # noqa: E731
    rho = 1 + 0.3 * np.sin(x + 1) * np.cos(y) * np.cos(z + 2) + noise()
    v = [0.1 * np.sin(x) * np.cos(y + 1) + noise(), 0.4 + 0.1 * np.cos(y + 2) + noise(), 0.1 * np.sin(z + y) + noise()]
    p = 2.5 + 0.2 * np.cos(x) * np.cos(y)
    U = to_fp32(np.stack([rho] + [rho * q for q in v] + [p / 0.4 + 0.5 * rho * sum(q * q for q in v)]))
    prm = {"heat_capacity_ratio": 1.4, "dynamic_viscosity": mu, "gravitational_acceleration": [0.0, 0.0, -0.1 if coords == "cartesian" else 0.0]}
    if coords == "cartesian":
        kinds = [["neumann"] * 4 + ["periodic"] * 2] * 5
    else:
        kinds = [(["reflecting"] if q == 1 else ["neumann"]) * 2 + ["periodic"] * 4 for q in range(5)]
    sim = Simulation("navier_stokes", coords, cfg, prm,
                     {"reconstructor": reconstructors.muscl, "slope_limiter": getattr(slope_limiters, limiter),
                      "riemann_solver": riemann_solvers.hll},
                     bcs_dict("navier_stokes", kinds), time_integrators.rk3_ssp, precision="fp32")
    sim.upload(U)
    sim.step(steps, dt=dt)
    assert sim.status() == 0
    got = sim.download()
    sim.close()
    O.run("navier_stokes", U, prm, O.Geometry(coords, cfg),
          dict(reconstructor="muscl", slope_limiter=limiter, riemann_solver="hll"), oracle_bcs(kinds), "rk3_ssp", 0.4,
          steps, dt_fixed=dt)
    I3 = (slice(None),) + (slice(1, -1),) * 3
    return float(np.linalg.norm(got[I3] - U[I3]) / np.linalg.norm(U[I3]))


def test_cartesian():
    assert error("cartesian", (64, 64, 64), (0, 0, 0), (1, 1, 1), 0.0, "minmod", 5, 2.0 ** -10) <= 3.8525e-8


ANNULUS = ((96, 128, 8), (0.5, 0, 0), (1.5, 2 * np.pi, 0.125))
SHELL = ((96, 64, 16), (0.5, 0.25 * np.pi, 0), (1.5, 0.75 * np.pi, 0.4))


@pytest.mark.parametrize("coords,grid,mu,before",
                         [("cylindrical", ANNULUS, 0.0, 5.0740e-8), ("cylindrical", ANNULUS, 1e-4, 5.1096e-8),
                          ("spherical", SHELL, 0.0, 5.1520e-8), ("spherical", SHELL, 1e-4, 5.1562e-8)])
def test_curvilinear(coords, grid, mu, before):
    assert error(coords, *grid, mu, "van_leer", 10, 2.0 ** -10) <= before
