"""The shared-memory-free step where its launches (programmatic dependent ones)
meet something else: the legacy stream, a captured graph, kernels of another
library between two steps, and a device without room for its scratch.  Each
against a handle with pinned z-marching kernels, bit for bit."""
import numpy as np
import pytest

import lbman3d_b200 as L
from lbman3d_b200 import _native as N

pytestmark = pytest.mark.gpu

GRID = (20, 18, 13)


def _pair(precision, grid=GRID):
    nx, ny, nz = grid
    p = L.Params(nx=nx, ny=ny, nz=nz, ALPHA=0.02)
    rng = np.random.default_rng(4)
    state = (1.0 + 0.01 * rng.standard_normal(p.V), 0.005 * rng.standard_normal(3 * p.V),
             0.1 * rng.standard_normal(5 * p.V))
    sims = [L.Simulation(p, L.ChannelConfig(), precision),
            L.Simulation(p, L.ChannelConfig(), precision, N.KERNELS_SPLIT, tile=(14, 14, 4))]
    for s in sims:
        s.upload(*state)
    return sims


def _same(a, b):
    x, y = a.download(f=True, force=True), b.download(f=True, force=True)
    for k in x:
        np.testing.assert_array_equal(x[k], y[k], err_msg=k)


PREC = pytest.mark.parametrize("precision", [L.Precision.FP64, L.Precision.FP16], ids=["fp64", "fp16"])


@PREC
def test_legacy_stream_with_other_kernels_between(precision):
    import torch
    a, b = _pair(precision)
    a.set_stream(0)
    x = torch.zeros(1 << 20, device="cuda")
    for n in (1, 3, 2):
        x += 1
        a.step(n)
        x *= 2
        b.step(n)
    _same(a, b)
    for s in (a, b):
        s.close()


@PREC
def test_captured_steps(precision):
    import torch
    a, b = _pair(precision)
    st = torch.cuda.Stream()
    a.set_stream(st.cuda_stream)
    a.step(2)
    a.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=st):
        a.step(2)
    with torch.cuda.stream(st):
        for _ in range(3):
            g.replay()
    st.synchronize()
    for _ in range(4):
        b.step(2)
    _same(a, b)
    g.reset()
    for s in (a, b):
        s.close()


def test_without_room_for_the_scratch():
    import torch
    word = 128 ** 3 * 4  # bytes of one FP32 field component: 8 MB
    torch.cuda.synchronize()
    probe = L.Simulation(L.Params(nx=8, ny=8, nz=8), L.FullyPeriodicConfig(), L.Precision.FP32)  # loads the module
    probe.init_seeded(1, 0.5, 1e-3)
    probe.step(1)
    probe.close()
    # 37 words of fields and staging; the point kernels want 57 free after the first 31
    hog = torch.empty(torch.cuda.mem_get_info()[0] - 45 * word, dtype=torch.uint8, device="cuda")
    before = torch.cuda.mem_get_info()[0]
    tight = L.Simulation(L.Params(nx=128, ny=128, nz=128), L.FullyPeriodicConfig(), L.Precision.FP32)
    used = before - torch.cuda.mem_get_info()[0]
    del hog
    torch.cuda.empty_cache()
    roomy = L.Simulation(L.Params(nx=128, ny=128, nz=128), L.FullyPeriodicConfig(), L.Precision.FP32)
    for s in (tight, roomy):
        s.init_seeded(3, 0.5, 1e-3)
        s.step(3)
    _same(tight, roomy)
    assert used < (37 + 5) * word  # without the 9 words of scratch
    for s in (tight, roomy):
        s.close()


@pytest.mark.parametrize("precision", [L.Precision.FP64, L.Precision.FP32], ids=["fp64", "fp32"])
@pytest.mark.parametrize("grid", [(24, 20, 16), (25, 22, 18), (17, 13, 11)], ids=["aligned", "odd_x", "primes"])
def test_transforms_leave_the_fields(grid, precision):
    """The spectrum and the correlation transform the handle's own u and Q."""
    nx, ny, nz = grid
    rng = np.random.default_rng(nx)
    with L.Simulation(L.Params(nx=nx, ny=ny, nz=nz), L.FullyPeriodicConfig(), precision) as s:
        V = nx * ny * nz
        s.upload(1.0 + 0.01 * rng.standard_normal(V), 0.005 * rng.standard_normal(3 * V), 0.1 * rng.standard_normal(5 * V))
        s.step(1)
        x = s.download(f=True)
        s.velocity_spectrum()
        s.q_correlation()
        s.statistics()
        y = s.download(f=True)
    for k in x:
        np.testing.assert_array_equal(x[k], y[k], err_msg=k)
