"""Handles of one kind made and stepped from several threads: preparing a kernel
for one handle never disturbs the launches of another (its shared-memory limit
does not shrink for a moment, and its resident blocks are published whole)."""
import threading

import numpy as np
import pytest

from tests.helpers import bcs_dict, random_ns_state, to_fp32

pytestmark = pytest.mark.gpu

KINDS = [("navier_stokes", 0.0), ("navier_stokes", 1e-3), ("maxwell", None)]


def _make(physics, mu):
    from multiphysics_fvm_b200.backend import Simulation
    from multiphysics_fvm_b200.numerics import reconstructors, riemann_solvers, slope_limiters, time_integrators
    prm = ({"heat_capacity_ratio": 1.4, "dynamic_viscosity": mu, "gravitational_acceleration": [0, 0, 0]}
           if physics == "navier_stokes" else
           {"magnetic_permeability": 1.0, "electric_permittivity": 1.0, "electrical_conductivity": 0.0,
            "charge_density": 0.0, "magnetic_cleaning_coeff": 0.001, "electric_cleaning_coeff": 0.001})
    cfg = dict(x1_min=0.5, x1_max=1.5, x2_min=0.6, x2_max=1.4, x3_min=0, x3_max=0.6, nx1=33, nx2=9, nx3=4)
    return Simulation(physics, "cylindrical", cfg, prm,
                      {"reconstructor": reconstructors.muscl, "slope_limiter": slope_limiters.monotonized_central,
                       "riemann_solver": riemann_solvers.rusanov},
                      bcs_dict(physics, [["neumann", "neumann"] + ["periodic"] * 4] * (5 if mu is not None else 6)),
                      time_integrators.rk3, precision="fp32")


@pytest.mark.parametrize("physics,mu", KINDS)
def test_prepare_and_launch_from_many_threads(physics, mu):
    shape = (35, 11, 6)
    rng = np.random.default_rng(3)
    U = to_fp32(random_ns_state(shape, rng) if physics == "navier_stokes" else rng.uniform(-1, 1, (6,) + shape))
    outs, errors, start = [], [], threading.Barrier(8)

    def work():
        try:
            start.wait()
            for _ in range(60):
                sim = _make(physics, mu)
                sim.upload(U)
                r = sim.residual()
                sim.upload(U)
                sim.step(2, dt=1e-4)
                assert sim.status() == 0
                outs.append((r, sim.download()))
                sim.close()
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    pool = [threading.Thread(target=work) for _ in range(8)]
    for t in pool:
        t.start()
    for t in pool:
        t.join()
    assert not errors, errors[0]
    assert len(outs) == 8 * 60
    for r, u in outs[1:]:
        assert np.array_equal(r, outs[0][0]) and np.array_equal(u, outs[0][1])
