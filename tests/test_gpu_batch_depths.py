"""Batches whose descriptors ask for different z-march depths (fvm_desc.zchunk;
0 is the default split): the depth decides only which block computes a cell, so
every grid's state is bitwise that of the batch with depth 0 throughout.  One
group per kernel that takes tile lists: the mixed launch, the float32 list
kernels (two limiters keep the grids out of the mixed launch), float64."""
import ctypes as C
import math

import numpy as np
import pytest

from tests.helpers import bcs_dict, random_ns_state, to_fp32

pytestmark = pytest.mark.gpu

HEAT = {"mass_density": 1.0, "specific_heat_capacity": 1.0, "thermal_conductivity": 1.0, "volumetric_heat_source": 0.1}
NS = {"heat_capacity_ratio": 1.4, "dynamic_viscosity": 0.0, "gravitational_acceleration": [0.0, 0.1, -0.2]}
# (physics, (nx1, nx2, nx3), limiter; None: piecewise constant)
GROUPS = {
    "mixed": ("fp32", [("navier_stokes", (64, 40, 48), "minmod"), ("heat", (40, 50, 37), None),
                       ("navier_stokes", (70, 64, 1), "minmod"), ("heat", (33, 24, 20), None)]),
    "list": ("fp32", [("navier_stokes", (48, 40, 48), "minmod"), ("navier_stokes", (40, 33, 37), "minmod"),
                      ("navier_stokes", (33, 24, 20), "van_leer"), ("heat", (40, 24, 35), None),
                      ("heat", (24, 40, 20), None)]),
    "float64": ("fp64", [("navier_stokes", (48, 40, 48), "minmod"), ("navier_stokes", (40, 33, 37), "minmod"),
                         ("navier_stokes", (64, 48, 1), "minmod")]),
}


def _batch(precision, grids, depths):
    from multiphysics_fvm_b200 import _lib as L
    from multiphysics_fvm_b200.backend import Batch, Simulation
    from multiphysics_fvm_b200.numerics import reconstructors, riemann_solvers, slope_limiters, time_integrators
    lib = L.load()
    b = Batch.__new__(Batch)
    b.sims, b._lib, b._b = [], lib, C.c_void_p()
    descs = (L.FvmDesc * len(grids))()
    for i, (physics, n, lim) in enumerate(grids):
        sim = Simulation.__new__(Simulation)
        cfg = dict(x1_min=0, x1_max=1, x2_min=0, x2_max=0.9, x3_min=0, x3_max=1.1, nx1=n[0], nx2=n[1], nx3=n[2])
        schemes = {"riemann_solver": riemann_solvers.hll,
                   "reconstructor": reconstructors.muscl if lim else reconstructors.piecewise_constant,
                   "slope_limiter": getattr(slope_limiters, lim or "minmod")}
        nv = 5 if physics == "navier_stokes" else 1
        bcs = bcs_dict(physics, [["neumann", "neumann"] + ["periodic"] * 4] * nv)
        descs[i] = sim._describe(physics, "cartesian", cfg, NS if nv == 5 else HEAT, schemes, bcs,
                                 time_integrators.rk3, precision, depths[i % len(depths)], 0)
        b.sims.append(sim)
    L.check(lib.fvm_batch_create(descs, len(grids), C.byref(b._b)), "fvm_batch_create")
    for i, sim in enumerate(b.sims):
        h = C.c_void_p()
        L.check(lib.fvm_batch_handle(b._b, i, C.byref(h)), "fvm_batch_handle")
        sim._attach(h, lib, owned=False)
    return b


def _run(precision, grids, depths):
    b = _batch(precision, grids, depths)
    rng = np.random.default_rng(4)
    for sim, (physics, n, _) in zip(b.sims, grids):
        shape = tuple(x + 2 for x in n)
        U = random_ns_state(shape, rng) if physics == "navier_stokes" else rng.uniform(1.0, 2.0, (1,) + shape)
        sim.upload(to_fp32(U))
        sim.set_time(0.0, math.inf, 0.2)
    b.step(2)
    assert all(sim.status() == 0 for sim in b.sims)
    out = [sim.download() for sim in b.sims]
    b.close()
    return out


@pytest.mark.parametrize("depths", [(0, 16), (16, 0), (0, 0, 7), (5, 64)], ids=lambda d: "d" + "_".join(map(str, d)))
@pytest.mark.parametrize("group", list(GROUPS))
def test_depths_of_members_may_differ(group, depths):
    precision, grids = GROUPS[group]
    for got, ref in zip(_run(precision, grids, depths), _run(precision, grids, (0,))):
        assert np.array_equal(got, ref)
