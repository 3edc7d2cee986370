"""Diagnostics kernels at the edges of their tiles (energy 32 x 8 columns, defects
31 x 15, marches of 2 to 32 planes, flow sums two cells per turn) against the
oracle on the values the device holds, so only FP64 rounding separates them."""
import numpy as np
import pytest

import lbman3d_b200 as L
from lbman3d_b200 import _native as N
from oracle import oracle as O

pytestmark = pytest.mark.gpu

GRIDS = [(2, 2, 2), (3, 17, 5), (31, 15, 4), (32, 16, 3), (33, 8, 7), (63, 9, 2), (30, 31, 33), (1, 40, 6)]


@pytest.mark.parametrize("precision", [L.Precision.FP64, L.Precision.FP32], ids=["fp64", "fp32"])
@pytest.mark.parametrize("bc", ["periodic", "channel", "box_mixed"])
@pytest.mark.parametrize("grid", GRIDS, ids=["x".join(map(str, g)) for g in GRIDS])
def test_sums_and_defects_at_tile_edges(grid, bc, precision):
    from cases import BC
    nx, ny, nz = grid
    V = nx * ny * nz
    rng = np.random.default_rng(V)
    sim = L.Simulation(L.Params(nx=nx, ny=ny, nz=nz), L.from_face_tuples(BC[bc]), precision)
    sim.upload(1 + 0.01 * rng.standard_normal(V), 0.01 * rng.standard_normal(3 * V), 0.2 * rng.standard_normal(5 * V))
    d = sim.reduce(N.DIAG_ALL)
    have = sim.download()
    sim.close()
    p = O.make_params(nx, ny, nz, BC[bc])
    lg = O.log_reduce(p, have["rho"], have["u"], np.zeros(3 * V))
    absu = np.abs(have["u"]).reshape(3, V)
    scale = [V, *(have["rho"].ravel() * absu).sum(axis=1), *lg[4:8]]
    # V terms of either sign, each to a few 2^-53: far below 1e-12 of the sum of their magnitudes
    for k, key in enumerate(("mass", "px", "py", "pz", "kinetic_energy", "rel_change_num", "rel_change_den", "umax2")):
        assert abs(d[key] - lg[k]) <= 1e-12 * scale[k], key
    fe = O.free_energy(p, have["q"])
    assert abs(d["free_energy"] - fe) <= 1e-11 * (abs(fe) + V * 0.2 ** 2 * p.L)
    if min(grid) >= 2:
        # FP32 directors are rounded: a face may turn where a dot product is below
        # 1e-7, about one in 10^5 of these random faces
        n = O.winding(p, O.order_director(p, have["q"])[1])[0]
        assert abs(d["defect_faces"] - n) <= (0 if precision == L.Precision.FP64 else 2)
    else:
        assert d["defect_faces"] == -1


# 8-column and 16-row descriptor tiles, marches of one and two planes, and
# marches with a short last range
@pytest.mark.parametrize("grid", [(8, 16, 1), (8, 16, 2), (24, 32, 21)])
def test_closure_marches_at_their_edges(grid):
    from lbman3d_b200 import closure as CL
    from oracle import closure as K
    V = grid[0] * grid[1] * grid[2]
    r = np.random.default_rng(V)
    feat, tgt = r.standard_normal((9, V)).astype(np.float32), r.standard_normal((8, V)).astype(np.float32)
    feat[0] += 1.0
    with CL.Closure(*grid, seed=6) as cl:
        prm = cl.params()
        sh, sc, osc = cl.scales()
        got = cl.forward(feat)
        loss, g = cl.gradient(feat, tgt)
    ref = K.forward(feat, grid, prm, sh, sc, bf=True)[0][..., :8].reshape(-1, 8).T
    assert np.max(np.abs(got - ref)) <= 2e-2 * np.max(np.abs(ref))  # bf16 activations: a few 2^-8
    lref, gref = K.loss_and_grad(feat, tgt, grid, prm, sh, sc, osc, bf=True)
    assert abs(loss - lref) <= 1e-3 * lref
    for (w0, b0), (_, cout) in zip(K.OFFSETS, K.LAYERS):
        for a, b in ((w0, b0), (b0, b0 + cout)):
            x, y = g[a:b].astype(np.float64), gref[a:b]
            assert np.linalg.norm(x - y) <= 3e-2 * max(np.linalg.norm(y), 1e-30), (a, b)
