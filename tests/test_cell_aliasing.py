"""The in-place LBM cell functions write the velocity array that a force formed on
the fly reads (PointForce's -MU u, the cell's own value), so they may not claim,
by __restrict__, that nothing else reads it."""
import os
import re

import pytest

LBM = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "lbman3d_b200", "csrc", "lbm.cuh")


@pytest.mark.parametrize("fn", ["aa_even_cell", "aa_odd_cell", "aa_even_h2", "aa_odd_h2"])
def test_velocity_is_not_restrict(fn):
    with open(LBM) as fh:
        params = re.search(r"__forceinline__ void " + fn + r"\((.*?)\)\s*\{", fh.read(), re.S).group(1)
    assert re.search(r"\*\s*uout\b", params) and not re.search(r"__restrict__\s+uout\b", params)
