"""Kernels that overlap their set-up with the kernel before them: where tensor
memory is allocated in relation to the hand-over.

An allocation waits until the columns are free.  A later kernel's CTA that holds
columns while it waits for an earlier kernel must therefore not be launched before
that kernel has allocated: the hand-over (pdl_go) comes after the allocation, or
the allocation after the wait (pdl_wait), when nothing is waited for any more.
Read from the kernels' source."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "chymera_uo_b200", "csrc")


def kernels():
    """(file, kernel, body) of every __global__ function that overlaps."""
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        text = re.sub(r"//[^\n]*", "", open(path).read())
        # the helper that allocates on a kernel's behalf
        text = text.replace("wide_setup(c, sm, t, x);", "tcgen05.alloc")
        for m in re.finditer(r"__global__ void (?:__launch_bounds__\([^)]*\) )?(\w+)\(", text):
            start = text.index("{", text.index(")", m.end()))
            depth, i = 0, start
            while True:
                depth += {"{": 1, "}": -1}.get(text[i], 0)
                i += 1
                if depth == 0:
                    break
            body = text[start:i]
            if "pdl_wait()" in body and "tcgen05.alloc" in body:
                yield os.path.basename(path), m.group(1), body


FOUND = list(kernels())


def test_the_kernels_are_found():
    assert {k for _, k, _ in FOUND} == {"k_mode_mixed", "k_wide_down", "k_wide_up", "k_wide_sweep_tm", "k_thomas_tm",
                                        "k_blk_solve_tab"}


@pytest.mark.parametrize("file,kernel,body", FOUND, ids=[k for _, k, _ in FOUND])
def test_allocation_before_hand_over_or_after_wait(file, kernel, body):
    alloc, go, wait = body.index("tcgen05.alloc"), body.index("pdl_go()"), body.index("pdl_wait()")
    assert alloc < go or wait < alloc, (file, kernel)
