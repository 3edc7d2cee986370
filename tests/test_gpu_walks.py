"""Walks of 2, 4 and 8 planes of the packed point update on planes of 2^15 cells
and more, each with a short last chunk, upwind and between x and y walls: the
chunk edges, where the force's z terms are left to its reader, against the
z-marching kernels bit for bit."""
import numpy as np
import pytest

import lbman3d_b200 as L
from lbman3d_b200 import _native as N

pytestmark = pytest.mark.gpu


# 150 blocks per chunk, 888 wanted on 148 SMs: 11, 23 and 57 planes walk 2, 4 and 8
@pytest.mark.parametrize("nz,bc,upwind,precision", [
    (11, "channel", True, L.Precision.FP32), (23, "periodic", True, L.Precision.FP32),
    (57, "channel", False, L.Precision.FP32), (57, "box_mixed", True, L.Precision.FP32),
    (23, "channel", True, L.Precision.FP16), (57, "periodic", True, L.Precision.FP16)])
def test_short_walks_on_wide_planes(nz, bc, upwind, precision):
    from cases import BC
    p = L.Params(nx=240, ny=160, nz=nz, ALPHA=0.02, MU=0.01,
                 kQAdvection=L.Advection.Upwind if upwind else L.Advection.Centred)
    rng = np.random.default_rng(nz)
    state = (1.0 + 0.01 * rng.standard_normal(p.V), 0.005 * rng.standard_normal(3 * p.V),
             0.1 * rng.standard_normal(5 * p.V))
    out = []
    for kernels, tile in ((N.KERNELS_AUTO, None), (N.KERNELS_SPLIT_PAIR, (30, 10, 32))):
        with L.Simulation(p, L.from_face_tuples(BC[bc]), precision, kernels, tile=tile) as s:
            s.upload(*state)
            s.step(1)
            s.step(2)
            s.qtensor_step()
            s.lbm_step()
            out.append(s.download(force=True))
    for k in out[0]:
        np.testing.assert_array_equal(out[0][k], out[1][k], err_msg=k)


def test_fp64_force_in_a_kernel_of_its_own():
    """FP64 boxes of more than 6 M cells with walls of every kind."""
    from cases import BC
    p = L.Params(nx=186, ny=187, nz=185, ALPHA=0.02, MU=0.01)
    rng = np.random.default_rng(8)
    state = (1.0 + 0.01 * rng.standard_normal(p.V), 0.005 * rng.standard_normal(3 * p.V),
             0.1 * rng.standard_normal(5 * p.V))
    out = []
    for kernels, tile in ((N.KERNELS_AUTO, None), (N.KERNELS_SPLIT, (14, 14, 32))):
        with L.Simulation(p, L.from_face_tuples(BC["box_mixed"]), L.Precision.FP64, kernels, tile=tile) as s:
            s.upload(*state)
            s.step(1)
            s.step(2)
            out.append(s.download(force=True))
    for k in out[0]:
        np.testing.assert_array_equal(out[0][k], out[1][k], err_msg=k)
