"""FP32 trajectories and flow steps with rectangles on pairs of sites (site
map 6) against the scalar two-row form (site map 3): each direction paired,
the smallest extents, partly filled blocks, both integrators with odd and even
step counts, re-unitarisation on and off, and lattices that cannot be paired."""

import numpy as np
import pytest

# the last direction of even extent >= 4 is paired -- t (two of 4 sites, 16384 pairs; a partly filled last block;
# extents of 1 to 3 beside it), z, y, x -- or none
SHAPES = [(32, 16, 16, 4), (13, 11, 9, 26), (3, 1, 2, 6000), (17, 15, 26, 5), (19, 36, 7, 7), (64, 7, 9, 9),
          (33, 31, 33, 1)]


def pair_variant(q):
    return next(i for i, v in enumerate(q.force_variants()) if v["site_map"] == 6)


@pytest.fixture
def both(q):
    """Run f() with the paired and with the scalar shape."""
    old = q.force_get_variant(q.F32, True)

    def run(f):
        out = []
        for v in (pair_variant(q), 10):
            q.force_set_variant(q.F32, True, v)
            out.append(f())
        return out

    yield run
    q.force_set_variant(q.F32, True, old)


def start(q, ts):
    gf = q.GaugeField(q.Geometry(ts))
    gf.set_rand(q.RngState("pairs").split("gf"), 0.3, 1)
    gm = q.GaugeMomentum(gf.geo)
    gm.set_rand(q.RngState("pairs").split("gm"), 1.0)
    return gf, gm


# FP32: a step's force sums 18 staples of 3-4 products (2e-6 relative, as the single force's own test), some ten steps
TOL = 2e-5


@pytest.mark.gpu
@pytest.mark.parametrize("ts", SHAPES)
@pytest.mark.parametrize("integrator,n_step", [("force-gradient", 3), ("leapfrog", 4), ("leapfrog", 5)])
@pytest.mark.parametrize("reunit", [0, 2])
def test_trajectory(q, both, ts, integrator, n_step, reunit):
    gf, gm = start(q, ts)
    ga = q.GaugeAction(2.13, -0.331)

    def traj():
        for _ in range(2):  # direct, then the recorded graph
            u, p = gf.copy(), gm.copy()
            dh = q.run_hmc_evolve_pure_gauge(p, u, ga, None, n_step, integrator=integrator, precision="mixed",
                                             reunit_interval=reunit)
        return np.asarray(u), np.asarray(p), dh

    (u, p, dh), (u2, p2, dh2) = both(traj)
    assert np.abs(u - u2).max() < TOL and np.abs(p - p2).max() < 10 * TOL
    assert abs(dh - dh2) < 1e-4 * max(1.0, abs(dh2)) + 1e-6 * 24 * gf.geo.total_volume


@pytest.mark.gpu
@pytest.mark.parametrize("ts", SHAPES)
def test_flow_step(q, both, ts):
    gf, _ = start(q, ts)

    def flow():
        g = gf.copy(precision=q.F32)
        for _ in range(2):
            q.gf_wilson_flow_step(g, 0.02, c1=-0.331)
        return np.asarray(g)

    a, b = both(flow)
    assert np.abs(a - b).max() < TOL
    g64 = gf.copy()
    for _ in range(2):
        q.gf_wilson_flow_step(g64, 0.02, c1=-0.331)
    assert np.abs(a - np.asarray(g64)).max() < TOL


@pytest.mark.gpu
def test_autotuner_times_the_paired_shape(q):
    gf, _ = start(q, (16, 16, 16, 16))
    old = q.force_get_variant(q.F32, True)
    best, ms = q.autotune_force(gf.copy(precision=q.F32), -0.331, 1)
    assert 0 <= best < len(q.force_variants()) and ms > 0
    q.force_set_variant(q.F32, True, old)
