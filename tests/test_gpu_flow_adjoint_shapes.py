"""The plaquette flow's pull-back kernel against the general one (every path
as a product of dual matrices), which a rectangle coefficient of 1e-30
selects, on lattices of extents 1 to 3 and around the 128 sites of a block,
with su(3) and general cotangents."""

import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("ts", [(1, 2, 3, 4), (2, 2, 2, 2), (3, 5, 3, 3), (4, 4, 4, 2), (5, 3, 3, 3), (8, 4, 4, 3)])
@pytest.mark.parametrize("single", [False, True])
def test_plaquette_pull_back_matches_dual_matrices(q, ts, single):
    prec = q.F32 if single else q.F64
    geo = q.Geometry(ts)
    gf = q.GaugeField(geo)
    gf.set_rand(q.RngState("adjoint-shapes"), 0.3, 1)
    rng = np.random.default_rng(int(np.prod(ts)))
    lam = rng.standard_normal((gf.geo.total_volume, 4, 3, 3, 2)) @ [1, 1j]
    anti = (lam - np.conj(np.swapaxes(lam, -1, -2))) / 2
    anti -= np.trace(anti, axis1=-2, axis2=-1)[..., None, None] / 3 * np.eye(3)
    g = gf.copy(precision=prec)
    got = []
    for c1, cotangent in ((0.0, anti), (1e-30, anti), (0.0, lam)):
        c = q.GaugeMomentum(geo).from_numpy(cotangent).copy(precision=prec)
        got.append(np.asarray(q.gf_wilson_flow_vjp(g, 0.05, 3, c, c1=c1, checkpoint_every=2)))
    # nine stages of some 50 products each: 500 units of rounding
    tol = 500 * (6e-8 if single else 1.1e-16)
    n = np.linalg.norm(got[1])
    assert np.linalg.norm(got[0] - got[1]) < tol * n
    # a cotangent counts by its su(3) part
    assert np.linalg.norm(got[2] - got[0]) < tol * n
