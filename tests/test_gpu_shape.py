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


def test_the_own_shape_selects_the_point_kernels_again():
    """They keep scratch (seen as memory) and give the same bits before, while and
    after another shape is in use; a shape read back and set changes nothing."""
    p = L.Params(nx=100, ny=96, nz=97, ALPHA=0.02)
    rng = np.random.default_rng(2)
    state = (1.0 + 0.01 * rng.standard_normal(p.V), 0.005 * rng.standard_normal(3 * p.V),
             0.1 * rng.standard_normal(5 * p.V))
    scratch = 8 * 8 * p.V
    with L.Simulation(p, L.ChannelConfig(), L.Precision.FP64) as a, \
            L.Simulation(p, L.ChannelConfig(), L.Precision.FP64) as b:
        for s in (a, b):
            s.upload(*state)
        own = [a.shape()[k] for k in KEYS]
        free = _free()
        a.set_shape(*own)
        assert _free() == free
        for shape in (own, (N.KERNELS_SPLIT, 14, 14, 16), own):
            a.set_shape(*shape)
            a.step(3)
            b.step(3)
        assert _free() <= free and [a.shape()[k] for k in KEYS] == own
        a.set_shape(N.KERNELS_SPLIT, 14, 14, 16)
        assert _free() - free >= scratch
        x, y = a.download(f=True), b.download(f=True)
    for k in x:
        np.testing.assert_array_equal(x[k], y[k], err_msg=k)


def test_autotune_result_names_the_point_kernels():
    """32^3 FP64, where they are eight times as fast as any z march: the tuned
    shape is the handle's own, from any shape."""
    p = L.Params(nx=32, ny=32, nz=32)
    with L.Simulation(p, L.FullyPeriodicConfig(), L.Precision.FP64) as a:
        a.init_seeded(3, 0.5, 1e-3)
        own = [a.shape()[k] for k in KEYS]
        a.set_shape(N.KERNELS_SPLIT, 14, 14, 4)
        best = a.autotune(steps_per_trial=2)
        assert [best[k] for k in KEYS] == own == [a.shape()[k] for k in KEYS]
