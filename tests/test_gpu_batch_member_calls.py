"""Single-grid calls on the members of a batch that runs the tile-list kernels
(float32 grids outside the one-launch batch): residual, steps, timing and the
depth sweep run on a member as on a grid of its own.  The residual is held
against the float64 oracle (relative L-inf <= 2e-6, as for single grids), the
steps against the batch's own, which are bitwise the same, and the batch steps
on soundly after a member's sweep."""
import math

import numpy as np
import pytest

from oracle import fvm_oracle as O
from tests.helpers import bcs_dict, random_ns_state, rel_linf, to_fp32

pytestmark = pytest.mark.gpu

N = [(40, 24, 20), (33, 17, 9)]
KINDS = [["neumann", "neumann"] + ["periodic"] * 4] * 5


def _setups(coords, mu, limiters=("minmod", "van_leer")):
    from multiphysics_fvm_b200.numerics import reconstructors, riemann_solvers, slope_limiters, time_integrators
    from multiphysics_fvm_b200.physics import navier_stokes
    out = []
    for n, lim in zip(N, limiters):
        out.append({"physics": navier_stokes, "coordinate_system": coords,
                    "physical_parameters": {"heat_capacity_ratio": 1.4, "dynamic_viscosity": mu,
                                            "gravitational_acceleration": [0.0, 0.1, -0.2]},
                    "grid_config": dict(x1_min=1.0, x1_max=2.0, x2_min=0.6, x2_max=1.4, x3_min=0.0, x3_max=0.6,
                                        nx1=n[0], nx2=n[1], nx3=n[2]),
                    "time_integrator": time_integrators.rk3,
                    "space_schemes": {"riemann_solver": riemann_solvers.hll, "reconstructor": reconstructors.muscl,
                                      "slope_limiter": getattr(slope_limiters, lim)},
                    "boundary_conditions": bcs_dict("navier_stokes", KINDS), "precision": "fp32"})
    return out


@pytest.mark.parametrize("mu", [0.0, 1e-3], ids=["inviscid", "viscous"])
@pytest.mark.parametrize("coords", ["cartesian", "cylindrical", "spherical"])
def test_member_calls(coords, mu):
    from multiphysics_fvm_b200.backend import Batch
    setups = _setups(coords, mu)
    rng = np.random.default_rng(6)
    states = [to_fp32(random_ns_state(tuple(x + 2 for x in n), rng)) for n in N]

    def fresh():
        b = Batch(setups)
        for i, U in enumerate(states):
            b[i].upload(U)
            b[i].set_time(0.0, math.inf, 0.3)
        return b

    b = fresh()
    for i, (s, U) in enumerate(zip(setups, states)):
        ref = O.ns_rhs(U, O.Geometry(coords, s["grid_config"]), s["physical_parameters"],
                       dict(reconstructor="muscl", slope_limiter=("minmod", "van_leer")[i], riemann_solver="hll"))
        assert rel_linf(b[i].residual(), ref) <= 2e-6
        b[i].upload(U)
    b.step(3)
    by_batch = [b[i].download() for i in range(len(N))]
    b.close()

    b = fresh()
    for i in range(len(N)):
        b[i].step(3)
        assert b[i].status() == 0
        assert np.array_equal(b[i].download(), by_batch[i])
        assert b[i].time_steps(1) > 0 and b[i].profile_steps(1)[2] == 3
    b.close()


@pytest.mark.parametrize("mu", [0.0, 1e-3], ids=["inviscid", "viscous"])
@pytest.mark.parametrize("coords,limiters", [("cartesian", ("minmod", "van_leer")), ("cylindrical", ("minmod", "van_leer")),
                                             ("spherical", ("minmod", "van_leer")), ("cartesian", ("minmod", "minmod"))])
def test_member_autotune_keeps_the_kernels_shape(coords, limiters, mu):
    """Also on a member of the one-launch batch (the last case, inviscid)."""
    from multiphysics_fvm_b200.backend import Batch
    setups = _setups(coords, mu, limiters)
    rng = np.random.default_rng(6)
    states = [to_fp32(random_ns_state(tuple(x + 2 for x in n), rng)) for n in N]
    outs = []
    for tuned in (False, True):
        b = Batch(setups)
        rows = [b[i].tiling()[0] for i in range(len(N))]
        for i, U in enumerate(states):
            b[i].upload(U)
            b[i].set_time(0.0, math.inf, 0.3)
        if tuned:
            z, ms = b[0].autotune()
            assert z >= 1 and ms > 0 and [b[i].tiling()[0] for i in range(len(N))] == rows
            z, ms = b.autotune()  # rebuilds the batch's tables from its members
            assert z >= 1 and ms > 0
        b.step(2)
        assert all(b[i].status() == 0 for i in range(len(N)))
        outs.append([b[i].download() for i in range(len(N))])
        b.close()
    assert all(np.array_equal(x, y) for x, y in zip(*outs))
