"""The shared-memory-free time step (qpoint.cuh), which untuned AUTO handles
take: value for value the arithmetic of the z-marching kernels, so a box must
come out bit for bit as with explicitly chosen z-marching kernels, whole steps
and the Q stage alone, on every wall mask (none, x, x and y, all, anchoring,
mixed Q tags), on thin and odd boxes, and on boxes large enough for long walks."""
import numpy as np
import pytest

import lbman3d_b200 as L
from lbman3d_b200 import _native as N

pytestmark = pytest.mark.gpu


def _pair(grid, bc, precision, upwind, kernels, tile):
    """An AUTO handle and one with pinned z-marching kernels, same state."""
    from cases import BC
    nx, ny, nz = grid
    p = L.Params(nx=nx, ny=ny, nz=nz, ALPHA=0.02, MU=0.01,
                 kQAdvection=L.Advection.Upwind if upwind else L.Advection.Centred)
    rng = np.random.default_rng(nx + 7 * ny + 13 * nz)
    rho, u, q = (1.0 + 0.01 * rng.standard_normal(p.V), 0.005 * rng.standard_normal(3 * p.V),
                 0.1 * rng.standard_normal(5 * p.V))
    sims = [L.Simulation(p, L.from_face_tuples(BC[bc]), precision),
            L.Simulation(p, L.from_face_tuples(BC[bc]), precision, kernels, tile=tile)]
    for s in sims:
        s.upload(rho, u, q)
    return sims


def _same(a, b, f=True):
    x, y = a.download(f=f, force=True), b.download(f=f, force=True)
    for k in x:
        np.testing.assert_array_equal(x[k], y[k], err_msg=k)


# nx = 28 and 60 resolve to the packed pair arithmetic in FP32 / FP16 (30-wide
# tiles fit), the others to the one-point arithmetic
CASES = [((20, 18, 13), "periodic", False), ((20, 18, 13), "slit", True), ((33, 7, 10), "channel", False),
         ((9, 13, 11), "box_mixed", True), ((7, 6, 9), "qmixed", False), ((1, 5, 6), "box_mixed", False),
         ((130, 3, 2), "lid", True), ((28, 9, 11), "periodic", True), ((28, 30, 9), "channel", False),
         ((60, 5, 7), "box_mixed", True), ((28, 6, 1), "lid", False), ((60, 4, 8), "qper_uwall", False)]


@pytest.mark.parametrize("precision", [L.Precision.FP64, L.Precision.FP32, L.Precision.FP16],
                         ids=["fp64", "fp32", "fp16"])
@pytest.mark.parametrize("grid,bc,upwind", CASES, ids=[f"{'x'.join(map(str, c[0]))}-{c[1]}" for c in CASES])
def test_point_kernels_equal_the_marching_kernels_bitwise(grid, bc, upwind, precision):
    packed = grid[0] in (28, 60) and precision != L.Precision.FP64
    kernels, tile = (N.KERNELS_SPLIT_PAIR, (30, 6, 4)) if packed else (N.KERNELS_SPLIT, (14, 14, 4))
    a, b = _pair(grid, bc, precision, upwind, kernels, tile)
    for n in (1, 2, 4):  # odd and even in-place steps at the end of a call
        a.step(n)
        b.step(n)
        _same(a, b)
    for s in (a, b):  # the two halves of a step called apart
        s.qtensor_step()
    _same(a, b)
    for s in (a, b):
        s.lbm_step()
        s.step(1)
    _same(a, b)
    for s in (a, b):
        s.close()


# Large boxes, where a thread walks 4 planes (one point per thread) or 16 (packed,
# planes of 2^15 cells: the z terms of the force are finished in the walk, except
# at chunk boundaries), with a short last chunk.  FP64 there forms the force in a
# kernel of its own.
@pytest.mark.parametrize("grid,bc,precision", [((182, 187, 191), "box_mixed", L.Precision.FP32),
                                               ((240, 160, 165), "box_mixed", L.Precision.FP32),
                                               ((256, 240, 167), "periodic", L.Precision.FP32),
                                               ((256, 240, 167), "periodic", L.Precision.FP16),
                                               ((240, 160, 5), "slit", L.Precision.FP16),
                                               ((182, 187, 191), "periodic", L.Precision.FP64)],
                         ids=["one_point", "packed_mixed", "packed", "packed_fp16", "packed_thin_fp16", "fp64"])
def test_long_walks(grid, bc, precision):
    packed = grid[0] % 4 == 0
    a, b = _pair(grid, bc, precision, False, N.KERNELS_SPLIT_PAIR if packed else N.KERNELS_SPLIT,
                 (30, 10, 32) if packed else (14, 14, 32) if precision == L.Precision.FP64 else (32, 8, 32))
    for n in (1, 2):
        a.step(n)
        b.step(n)
        _same(a, b, f=False)
    for s in (a, b):
        s.qtensor_step()
    _same(a, b, f=False)
    for s in (a, b):
        s.close()
