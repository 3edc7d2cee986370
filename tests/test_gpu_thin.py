"""Boxes so tall that one thread block per few planes passes the 65535 blocks of
a launch's y or z dimension."""
import numpy as np
import pytest

import lbman3d_b200 as L
from lbman3d_b200 import _native as N

pytestmark = pytest.mark.gpu


def _state(V, seed=1):
    rng = np.random.default_rng(seed)
    return (1.0 + 0.01 * rng.standard_normal(V), 0.005 * rng.standard_normal(3 * V), 0.1 * rng.standard_normal(5 * V))


# 4 planes per thread would take 67501 chunks; nx = 28 takes the packed kernels
@pytest.mark.parametrize("grid,precision,kernels,tile", [
    ((4, 3, 270001), L.Precision.FP64, N.KERNELS_SPLIT, (14, 14, 32)),
    ((4, 3, 270001), L.Precision.FP32, N.KERNELS_SPLIT, (14, 14, 32)),
    ((28, 1, 270001), L.Precision.FP16, N.KERNELS_SPLIT_PAIR, (30, 6, 32))], ids=["fp64", "fp32", "packed_fp16"])
def test_point_kernels_step_a_tall_box(grid, precision, kernels, tile):
    nx, ny, nz = grid
    p = L.Params(nx=nx, ny=ny, nz=nz, ALPHA=0.02, MU=0.01)
    state, out = _state(p.V), []
    for k, t in ((N.KERNELS_AUTO, None), (kernels, tile)):
        with L.Simulation(p, L.SlitConfig(), precision, k, tile=t) as s:
            s.upload(*state)
            s.step(3)
            s.qtensor_step()
            s.lbm_step()
            out.append(s.download(force=True))
    for n in out[0]:
        np.testing.assert_array_equal(out[0][n], out[1][n], err_msg=n)


# more than 65535 of the 15-row tiles, of the 32-plane marches
@pytest.mark.parametrize("grid", [(2, 983100, 2), (2, 2, 2097200)], ids=["long_y", "tall"])
def test_defects_of_a_long_box(grid):
    from cases import BC
    from oracle import oracle as O
    nx, ny, nz = grid
    p = L.Params(nx=nx, ny=ny, nz=nz)
    with L.Simulation(p, L.FullyPeriodicConfig(), L.Precision.FP64) as s:
        s.upload(*_state(p.V))
        d = s.reduce(N.DIAG_DEFECTS)
        q = s.download()["q"]
    op = O.make_params(nx, ny, nz, BC["periodic"])
    assert d["defect_faces"] == O.winding(op, O.order_director(op, q)[1])[0]
