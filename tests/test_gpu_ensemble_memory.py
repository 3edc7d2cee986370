"""The two organisations of an ensemble each have buffers of their own (second
populations; stress): a stepped ensemble that changes between them keeps its
state, holds one kind at a time, and is created where only one kind fits."""
import numpy as np
import pytest

import lbman3d_b200 as L
from lbman3d_b200 import _native as N

pytestmark = pytest.mark.gpu


def _free():
    import torch
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def _boxes(sides, n):
    return [(L.Params(nx=s[0], ny=s[1], nz=s[2], ALPHA=0.01 + 0.002 * i, LAMBDA=0.3 + 0.1 * i),
             L.FullyPeriodicConfig() if i % 2 == 0 else L.SlitConfig()) for i, s in enumerate((sides * n)[:n])]


def _same(a, b, n):
    for i in range(n):
        x, y = a.download(i, f=True), b.download(i, f=True)
        for k in x:
            np.testing.assert_array_equal(x[k], y[k], err_msg=f"box {i} {k}")


@pytest.mark.parametrize("precision", [L.Precision.FP64, L.Precision.FP16], ids=["fp64", "fp16"])
def test_organisations_changed_under_way(precision):
    """SPLIT -> FUSED -> SPLIT after odd and even numbers of steps, through replayed
    graphs too, against an ensemble that stays as it is."""
    boxes = _boxes([(24, 18, 13), (16, 20, 9), (9, 13, 11)], 3)
    a, b = L.Ensemble(boxes, precision), L.Ensemble(boxes, precision)
    for e in (a, b):
        e.init_seeded(5)
    for kernels, steps in ((N.KERNELS_SPLIT, 3), (N.KERNELS_FUSED, 2), (N.KERNELS_SPLIT, 44), (N.KERNELS_FUSED, 45),
                           (N.KERNELS_FUSED, 1), (N.KERNELS_SPLIT, 1), (N.KERNELS_SPLIT, 0)):
        a.set_shape(kernels, 14, 14, 4)
        _same(a, b, len(boxes))  # a change of organisation alone changes nothing
        a.step(steps)
        b.step(steps)
        _same(a, b, len(boxes))
    for e in (a, b):
        e.close()


def test_a_change_of_organisation_gives_the_other_buffers_back():
    boxes = _boxes([(128, 128, 128)], 2)
    cells = sum(p.V for p, _ in boxes)
    e = L.Ensemble(boxes, L.Precision.FP32)
    e.init_seeded(1)
    split = _free()
    e.set_shape(N.KERNELS_FUSED, 14, 14, 16)
    # 15 words of populations for 9 of stress
    assert split - _free() <= (15 - 9) * 4 * cells + (4 << 20)
    e.set_shape(N.KERNELS_SPLIT, 14, 14, 16)
    assert split - _free() <= 4 << 20
    e.close()


def test_an_ensemble_without_room_for_the_stress():
    """FP16: 30 bytes per cell are left where the stress takes 36."""
    import torch
    boxes = _boxes([(128, 128, 128)], 4)
    out = []
    for tight in (False, True):
        hog = None
        if tight:  # 16 MB of staging and, per box, 220 MB of fields and 60 (stress: 72) MB more
            hog = torch.empty(_free() - ((16 + 4 * 220 + 265) << 20), dtype=torch.uint8, device="cuda")
        e = L.Ensemble(boxes, L.Precision.FP16)
        del hog
        torch.cuda.empty_cache()
        e.init_seeded(9)
        e.step(4)
        out.append((e.shape()["kernels"], e.download(0)))
        e.close()
    assert [k for k, _ in out] == [N.KERNELS_SPLIT, N.KERNELS_FUSED]
    for k in out[0][1]:
        np.testing.assert_array_equal(out[0][1][k], out[1][1][k], err_msg=k)
