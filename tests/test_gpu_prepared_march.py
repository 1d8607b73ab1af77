"""What a handle's first step prepares.  A kernel's shared-memory attribute is
set, and the kernel loaded, before the step's graph is captured, for every march
of the step: a three-dimensional grid's and a one-plane grid's.  Seen in the
CUDA calls of the first step of a fresh process."""
import json
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CHILD = """
import json, math, sys
import numpy as np, torch
from torch.profiler import ProfilerActivity, profile
from multiphysics_fvm_b200.backend import Simulation
from multiphysics_fvm_b200.numerics import reconstructors, riemann_solvers, slope_limiters, time_integrators
from tests.helpers import bcs_dict, random_ns_state
nx3, mu, precision, trace = int(sys.argv[1]), float(sys.argv[2]), sys.argv[3], sys.argv[4]
torch.zeros(1, device="cuda")
n = (40, 33, nx3)
cfg = dict(x1_min=0, x1_max=1, x2_min=0, x2_max=1, x3_min=0, x3_max=1, nx1=n[0], nx2=n[1], nx3=n[2])
sim = Simulation("navier_stokes", "cartesian", cfg,
                 {"heat_capacity_ratio": 1.4, "dynamic_viscosity": mu, "gravitational_acceleration": [0, 0, 0]},
                 {"reconstructor": reconstructors.muscl, "slope_limiter": slope_limiters.minmod,
                  "riemann_solver": riemann_solvers.hll},
                 bcs_dict("navier_stokes", [["periodic"] * 6] * 5), time_integrators.rk3_ssp, precision=precision)
sim.upload(random_ns_state(tuple(x + 2 for x in n), np.random.default_rng(1)))
sim.set_time(0.0, math.inf, 0.3)
with profile(activities=[ProfilerActivity.CPU, ProfilerActivity.CUDA]) as p:
    sim.step(1)
assert sim.status() == 0
p.export_chrome_trace(trace)
"""


@pytest.mark.parametrize("nx3,mu,precision", [(1, 0.0, "fp32"), (12, 0.0, "fp32"), (1, 1e-3, "fp32"), (1, 0.0, "fp64")])
def test_nothing_is_prepared_inside_the_capture(tmp_path, nx3, mu, precision):
    trace = tmp_path / "trace.json"
    r = subprocess.run([sys.executable, "-c", CHILD, str(nx3), str(mu), precision, str(trace)], cwd=ROOT,
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    calls = sorted((float(e["ts"]), e["name"]) for e in json.load(open(trace))["traceEvents"]
                   if e.get("cat") in ("cuda_runtime", "cuda_driver") and "ts" in e)
    at = {name: [t for t, c in calls if c.startswith(name)] for name in
          ("cudaStreamBeginCapture", "cudaStreamEndCapture", "cudaFuncSetAttribute")}
    assert len(at["cudaStreamBeginCapture"]) == 1 and len(at["cudaStreamEndCapture"]) == 1
    assert at["cudaFuncSetAttribute"], "the step's kernel was prepared"
    begin, end = at["cudaStreamBeginCapture"][0], at["cudaStreamEndCapture"][0]
    assert all(t < begin or t > end for t in at["cudaFuncSetAttribute"])
