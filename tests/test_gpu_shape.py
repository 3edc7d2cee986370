"""Launch shapes of an AUTO handle that steps with the shared-memory-free kernels:
it names them by the shape it was created with, and any other shape gives their
scratch (9 words per cell in FP32, 8 in FP64) back."""
import numpy as np
import pytest

import lbman3d_b200 as L
from lbman3d_b200 import _native as N

pytestmark = pytest.mark.gpu

KEYS = ("kernels", "tile_x", "tile_y", "zchunk")


def _free():
    import torch
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


@pytest.mark.parametrize("precision,words", [(L.Precision.FP64, 8), (L.Precision.FP32, 9)], ids=["fp64", "fp32"])
def test_another_shape_gives_the_scratch_back(precision, words):
    p = L.Params(nx=128, ny=128, nz=128)
    scratch = words * p.V * (8 if precision == L.Precision.FP64 else 4)
    with L.Simulation(p, L.FullyPeriodicConfig(), precision) as s:
        before = _free()
        s.set_shape(N.KERNELS_SPLIT, 14, 14, 16)
        assert _free() - before >= scratch
