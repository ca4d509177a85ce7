"""What a launch of the chain may read through the read-only path, by the source.

The blocks of a chained step may be there before the launch before it has made
its last write (chain_launch.cuh), so the pointers to what that launch may write,
the state and the accumulated forces, are not declared __restrict__ const: the
compiler would load them as data that stays as it is from the kernel's first
block on.
"""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "feriphys_gb300", "csrc")
CHAINED = [("step_grid.cu", "tile_step"), ("step_grid.cu", "k_step_grid_tiled"), ("step_general.cu", "k_step_general"),
           ("step_general.cu", "k_step_split"), ("step_general.cu", "k_terms64"), ("step_general.cu", "k_gather64")]


@pytest.mark.parametrize("source,name", CHAINED)
def test_state_pointers_of_chained_kernels_are_ordinary(source, name):
    text = open(os.path.join(CSRC, source)).read()
    m = re.search(r"\b%s\(([^)]*)\)\s*\{" % name, text)
    assert m, "definition of %s not found" % name
    read = [p for p in m.group(1).split(",") if re.search(r"\bconst\b.*\*.*\b(pos|vel|force_in)\s*$", p.strip())]
    assert len(read) >= 2, read
    assert not [p for p in read if "__restrict__" in p]
