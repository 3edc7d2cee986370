"""Boxes with FP16 populations sum the body force in one order on planes of any
size: a state with two periods in y steps, bit for bit, as the box of one period,
whose plane is below the size at which the packed FP32 kernels change theirs."""
import numpy as np
import pytest

import lbman3d_b200 as L
from lbman3d_b200 import _native as N

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kernels", [N.KERNELS_AUTO, N.KERNELS_SPLIT_PAIR], ids=["auto", "pair"])
@pytest.mark.parametrize("bc,nz", [("periodic", 37), ("slit", 5)])
def test_fp16_box_repeats_its_period(bc, nz, kernels):
    from cases import BC
    nx, ny = 240, 80  # 19200 and 38400 cells per plane, either side of 2^15
    rng = np.random.default_rng(nz)
    one = [1.0 + 0.01 * rng.standard_normal((1, nz, ny, nx)), 0.005 * rng.standard_normal((3, nz, ny, nx)),
           0.1 * rng.standard_normal((5, nz, ny, nx))]
    out = []
    for k in (1, 2):
        p = L.Params(nx=nx, ny=k * ny, nz=nz, ALPHA=0.02, MU=0.01)
        with L.Simulation(p, L.from_face_tuples(BC[bc]), L.Precision.FP16, kernels) as s:
            s.upload(*(np.tile(a, (1, 1, k, 1)).reshape(-1) for a in one))
            s.step(3)
            s.step(2)
            d = s.download(f=True)
        out.append({n: np.asarray(v).reshape(-1, nz, k * ny, nx) for n, v in d.items()})
    for n in out[0]:
        for h in range(2):
            np.testing.assert_array_equal(out[1][n][:, :, h * ny:(h + 1) * ny], out[0][n], err_msg=n)
