"""Order of the steps at the start of kernels that hold tensor memory, read from the source: a kernel may let its dependents start only when
it has its columns.  A dependent CTA that took them first would wait for a grid that waits for columns."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ai00_server_b200", "csrc")


def test_dependents_start_behind_the_allocation():
    seen = 0
    for f in sorted(os.listdir(CSRC)):
        if not f.endswith((".cu", ".cuh")) or f == "common.cuh":
            continue
        with open(os.path.join(CSRC, f)) as h:
            kernels = re.split(r"(?m)^__global__|^template <[^\n]*>\n__global__", h.read())[1:]
        for body in kernels:
            allocs, trigger = [m.start() for m in re.finditer(r"\btc_alloc2?\(", body)], body.find("pdl_launch_dependents()")      # (2: columns of a pair of SMs)
            if allocs and trigger >= 0:
                seen += 1
                assert max(allocs) < trigger, (f, body[:120])
    assert seen >= 5
