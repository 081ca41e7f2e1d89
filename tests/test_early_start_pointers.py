"""Kernels that start before the one ahead of them is complete (pdl_wait) read memory that another kernel
is still writing when they begin: no function that waits so may promise the compiler, by __restrict__,
that its pointers' memory has no other writer."""
import os
import re

from conftest import ROOT

SRC = os.path.join(ROOT, "afar_cudaeuler2dmixo3rk3solver_gb300", "csrc", "afar_kernels.cuh")


def test_no_restrict_in_functions_that_wait_for_the_kernel_ahead():
    # definitions end at a closing brace in the first column
    parts = re.split(r"(?m)^\}", open(SRC).read())
    waiting = [p for p in parts if re.search(r"\bpdl_wait\b\s*[<(]", p)]
    assert len(waiting) >= 4  # two reconstructs, the tile fetch and the stage tail
    for p in waiting:
        assert "__restrict__" not in p, p[:300]
