"""Rules that the kernel sources keep and no compiler checks."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "fuel_b200", "csrc")


def _kernels():
    for f in sorted(os.listdir(CSRC)):
        if f.endswith((".cu", ".cuh")):
            text = open(os.path.join(CSRC, f)).read()
            for m in re.finditer(r"__global__ void (?:__launch_bounds__\((?:[^()]|\([^()]*\))*\) )?(\w+)\(([^{;]*)\) \{\n(.*?)\n\}", text, re.S):
                yield f, m.group(1), m.group(2), m.group(3)


def test_nothing_read_after_the_wait_is_restrict():
    """A kernel that starts beside its predecessor waits before it reads what that one writes. A __restrict__ pointer would let
    the compiler take the load for one of constant data and move it above the wait. Kernels whose wait is their last statement
    read finished data only."""
    found = list(_kernels())
    assert len(found) > 40
    late = [name for _, name, _, body in found if body.rstrip().endswith("pdl_wait();")]
    assert "prefetch_l2_kernel" in late and "dequant_q4k_kernel" in late
    bad = [(f, name) for f, name, params, body in found
           if "__restrict__" in params and "pdl_wait()" in body and name not in late]
    assert not bad, bad
