"""Which memory the host transfers take: a device pointer in place of a host
array is refused with an error (in a child process, which an access to it from
the host would end), page-locked results are written by one copy, without the
staging ring."""
import ctypes as C
import json
import os
import subprocess
import sys

import numpy as np
import pytest

from tests.helpers import bcs_dict, random_ns_state

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
N = (24, 20, 16)


def make_sim():
    from multiphysics_fvm_b200.backend import Simulation
    from multiphysics_fvm_b200.numerics import reconstructors, riemann_solvers, slope_limiters, time_integrators
    cfg = dict(x1_min=0, x1_max=1, x2_min=0, x2_max=1, x3_min=0, x3_max=1, nx1=N[0], nx2=N[1], nx3=N[2])
    sim = Simulation("navier_stokes", "cartesian", cfg,
                     {"heat_capacity_ratio": 1.4, "dynamic_viscosity": 0.0, "gravitational_acceleration": [0, 0, 0]},
                     {"reconstructor": reconstructors.muscl, "slope_limiter": slope_limiters.minmod,
                      "riemann_solver": riemann_solvers.hll},
                     bcs_dict("navier_stokes", [["periodic"] * 6] * 5), time_integrators.rk3, precision="fp64")
    sim.upload(random_ns_state(tuple(x + 2 for x in N), np.random.default_rng(1)))
    return sim


DEVICE_POINTER = """
import ctypes as C, sys
import numpy as np, torch
from multiphysics_fvm_b200 import _lib as L
from tests.test_gpu_host_pointers import make_sim
sim = make_sim()
before = sim.download()
dev = torch.zeros(before.shape, dtype=torch.float64, device="cuda")
one = C.cast(dev.data_ptr(), C.POINTER(C.c_double))
per = (C.c_void_p * 5)(*[dev[q].data_ptr() for q in range(5)])
lib = L.load()
assert lib.fvm_upload(sim._h, one) != 0
assert lib.fvm_download(sim._h, one) != 0
assert lib.fvm_residual(sim._h, one) != 0
assert lib.fvm_upload_vars(sim._h, per) != 0
assert lib.fvm_download_vars(sim._h, per) != 0
assert np.array_equal(sim.download(), before) and not dev.any()
print("refused")
"""


def test_device_pointers_are_refused():
    r = subprocess.run([sys.executable, "-c", DEVICE_POINTER], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "refused" in r.stdout, (r.returncode, r.stderr[-2000:])


@pytest.mark.parametrize("call", ["upload", "download", "residual"])
def test_page_locked_arrays_are_copied_directly(tmp_path, call):
    import torch
    from torch.profiler import ProfilerActivity, profile
    from multiphysics_fvm_b200 import _lib as L
    sim, lib = make_sim(), L.load()
    want = sim.residual() if call == "residual" else sim.download()
    pinned = torch.empty(want.shape, dtype=torch.float64, pin_memory=True)
    if call == "upload":
        pinned.numpy()[...] = want
    ptr = C.cast(pinned.data_ptr(), C.POINTER(C.c_double))
    with profile(activities=[ProfilerActivity.CPU, ProfilerActivity.CUDA]) as p:
        L.check(getattr(lib, "fvm_" + call)(sim._h, ptr), call)
    p.export_chrome_trace(str(tmp_path / "trace.json"))
    copies = [e["name"] for e in json.load(open(tmp_path / "trace.json"))["traceEvents"]
              if e.get("cat") == "gpu_memcpy" and ("HtoD" in e["name"] or "DtoH" in e["name"])]
    assert len(copies) == 1
    assert np.array_equal(sim.download() if call == "upload" else pinned.numpy(), want)
