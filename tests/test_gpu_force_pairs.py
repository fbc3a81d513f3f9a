"""FP32 trajectories and flow steps with rectangles on pairs of sites (site
map 6) against the scalar two-row form (site map 3): both paired directions,
the smallest extents, partly filled blocks, both integrators with odd and even
step counts, re-unitarisation on and off; and the runs that stay scalar because
pairs would be slower, or the lattice cannot be paired."""

import numpy as np
import pytest

# t paired, or z where t is odd: three pairs along t, partly filled last blocks, extents of 1 to 3 beside the paired one
SHAPES = [(24, 24, 24, 6), (13, 11, 9, 26), (13, 11, 12, 26), (3, 1, 2, 6000), (3, 1, 6000, 3), (17, 15, 36, 5)]
# t of 4 sites (borders as large as the field), an even extent along y or x alone, none, few pairs
SCALAR = [(33, 31, 33, 4), (4, 25, 35, 35), (33, 4, 33, 9), (19, 36, 7, 7), (64, 7, 9, 9), (33, 31, 33, 1), (8, 8, 8, 8)]


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


def packed(q, f):
    """How many fields f() packs or unpacks."""
    q.prof_reset()
    q.prof_enable(True)
    try:
        f()
        q.synchronize()
        return q.prof_get("pair_pack")[1]
    finally:
        q.prof_enable(False)


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
@pytest.mark.parametrize("integrator,n_step", [("force-gradient", 8), ("leapfrog", 16), ("leapfrog", 17)])
@pytest.mark.parametrize("reunit", [0, 2])
def test_trajectory(q, both, ts, integrator, n_step, reunit):
    gf, gm = start(q, ts)
    ga = q.GaugeAction(2.13, -0.331)

    def once():
        u, p = gf.copy(), gm.copy()
        dh = q.run_hmc_evolve_pure_gauge(p, u, ga, None, n_step, integrator=integrator, precision="mixed",
                                         reunit_interval=reunit)
        return np.asarray(u), np.asarray(p), dh

    assert both(lambda: packed(q, once)) == [4, 0]  # links and momenta in and out
    # direct, then the recorded graph
    (u, p, dh), (u2, p2, dh2) = both(lambda: (once(), once())[1])
    assert np.abs(u - u2).max() < TOL and np.abs(p - p2).max() < 10 * TOL
    assert abs(dh - dh2) < 1e-4 * max(1.0, abs(dh2)) + 1e-6 * 24 * gf.geo.total_volume


@pytest.mark.gpu
@pytest.mark.parametrize("ts", SHAPES)
def test_flow_step(q, both, ts):
    gf, _ = start(q, ts)

    if ts[3] != 6:  # (three forces do not pay there)
        assert both(lambda: packed(q, lambda: q.gf_wilson_flow_step(gf.copy(precision=q.F32), 0.02, c1=-0.331))) == [2, 0]

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
@pytest.mark.parametrize("ts", SCALAR)
def test_runs_that_pairs_would_slow_stay_scalar(q, both, ts):
    gf, gm = start(q, ts)
    ga, g32 = q.GaugeAction(2.13, -0.331), gf.copy(precision=q.F32)

    def runs():
        for integrator in ("leapfrog", "force-gradient"):
            q.run_hmc_evolve_pure_gauge(gm.copy(), gf.copy(), ga, None, 8, integrator=integrator, precision="mixed")
        q.gf_wilson_flow_step(g32, 0.02, c1=-0.331)

    assert both(lambda: packed(q, runs)) == [0, 0]


@pytest.mark.gpu
def test_few_forces_do_not_pay_for_packing(q, both):
    gf, gm = start(q, (24, 24, 24, 24))
    ga = q.GaugeAction(2.13, -0.331)
    for n_step, fields in ((1, 0), (2, 0), (4, 4)):
        assert both(lambda: packed(q, lambda: q.run_hmc_evolve_pure_gauge(
            gm.copy(), gf.copy(), ga, None, n_step, integrator="leapfrog", precision="mixed"))) == [fields, 0]


@pytest.mark.gpu
def test_autotuner_times_the_paired_shape(q):
    gf, _ = start(q, (16, 16, 16, 16))
    old = q.force_get_variant(q.F32, True)
    best, ms = [], []
    n = packed(q, lambda: [x.append(y) for x, y in zip((best, ms), q.autotune_force(gf.copy(precision=q.F32), -0.331, 1))])
    assert n == 2  # its links and momenta, packed for the timing
    assert 0 <= best[0] < len(q.force_variants()) and ms[0] > 0
    q.force_set_variant(q.F32, True, old)


@pytest.mark.gpu
def test_packed_fields_are_given_back(q):
    ts = (16, 16, 16, 16)
    gf, gm = start(q, ts)
    ga = q.GaugeAction(2.13, -0.331)
    keep = []

    def traj():
        u, p = gf.copy(), gm.copy()
        keep.extend((u, p))  # (so that they do not go to the field pool)
        dh = q.run_hmc_evolve_pure_gauge(p, u, ga, None, 8, precision="mixed")
        return np.asarray(u), np.asarray(p), dh

    q.release_field_pool()
    want = [traj() for _ in range(3)][-1]
    # links, links, momenta: t of 8 + 4 pairs instead of 16 sites, two sites each
    assert q.release_field_pool() >= 3 * 4 * 16 ** 3 * 12 * 2 * 72
    for got in [traj() for _ in range(3)]:
        assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1]) and got[2] == want[2]
