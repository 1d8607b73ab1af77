"""A tensor-core kernel that gives up must wait for its MMAs and copies in flight
before it frees tensor memory.  Running out a wait with MMAs in flight is not
done on a GPU; this reads the kernels' source instead: the bounded wait that
ends a give-up is on a barrier that one commit (or one expected copy) completes
and no other role waits for, so that it is in phase 0 whatever had been done."""
import os
import re

import pytest

SRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "multiphysics_fvm_b200", "csrc",
                   "closure.cuh")


@pytest.mark.parametrize("kernel", ["conv3_kernel", "wgrad_kernel"])
def test_the_final_wait_is_on_a_barrier_of_its_own(kernel):
    text = open(SRC).read()
    start = re.search(r"__global__ void __launch_bounds__\([^;{]*?\) %s\(" % kernel, text).start()
    body = re.sub(r"//[^\n]*", "", text[start:text.index("\n}\n", start)])
    waits = re.findall(r"mbar_wait_bounded\((\w+), ([^,]+), WAIT_NS\)", body)
    assert "drain" in [bar for bar, _ in waits]
    for bar, parity in waits:
        assert parity.strip() == "0", f"{bar}: the phase depends on the path that led here"
        completes = re.findall(r"(?:umma_commit|mbar_arrive_expect_tx|mbar_arrive)\(%s\b" % bar, body)
        assert len(completes) == 1 and f"mbar_init({bar}, 1)" in body
    assert "role_wait(drain" not in body
    assert body.index("mbar_wait_bounded(drain") < body.index("tmem_dealloc(")
