"""The FP64 leapfrog with its link half steps fused into the force launch
against the composition gf_evolve(dt/2), gm += dt F, gf_evolve(dt/2) of single
operations, for odd and even step counts (the result in either of the two
link buffers), partly filled blocks, both force forms, and batches."""

import numpy as np
import pytest


def composed(q, gm, gf, ga, n_step):
    h0 = q.gm_hamilton_node(gm) + q.gf_hamilton_node(gf, ga)
    dt = 1.0 / n_step
    F = q.GaugeMomentum(gf.geo)
    for _ in range(n_step):
        q.gf_evolve(gf, gm, 0.5 * dt)
        q.set_gm_force(F, gf, ga)
        F *= dt
        gm += F
        q.gf_evolve(gf, gm, 0.5 * dt)
    q.unitarize(gf)
    return q.gm_hamilton_node(gm) + q.gf_hamilton_node(gf, ga) - h0


@pytest.mark.gpu
@pytest.mark.parametrize("ts", [(2, 2, 2, 2), (3, 3, 3, 5), (4, 4, 4, 4), (5, 4, 6, 7)])
@pytest.mark.parametrize("n_step", [1, 4, 5])
@pytest.mark.parametrize("c1", [0.0, -0.331])
def test_fused_leapfrog_matches_composition(q, ts, n_step, c1):
    geo, ga = q.Geometry(ts), q.GaugeAction(2.3, c1)
    gf = q.GaugeField(geo)
    gf.set_rand(q.RngState("leapfrog").split("gf"), 0.4, 1)
    gm = q.GaugeMomentum(geo)
    gm.set_rand(q.RngState("leapfrog").split("gm"), 1.0)
    gf2, gm2 = gf.copy(), gm.copy()
    for _ in range(2):  # direct, then through the recorded graph
        u, p = gf.copy(), gm.copy()
        dh = q.run_hmc_evolve_pure_gauge(p, u, ga, None, n_step, integrator="leapfrog")
    dh2 = composed(q, gm2, gf2, ga, n_step)
    # at most 5 steps, each some 100 operations on numbers of size 1
    assert np.abs(np.asarray(u) - np.asarray(gf2)).max() < 1e-13
    assert np.abs(np.asarray(p) - np.asarray(gm2)).max() < 1e-12
    assert abs(dh - dh2) < 1e-13 * 24 * geo.total_volume + 1e-12 * abs(dh2)
    # the same chain in a batch
    b = q.ChainBatch([ts, (4, 4, 4, 4)], [2.3, 5.5], [c1, 0.0])
    b.chain_from_numpy(0, np.asarray(gf))
    b.chain_from_numpy(1, np.asarray(q.GaugeField(q.Geometry((4, 4, 4, 4))).copy()) + np.eye(3))
    rs = q.RngState("leapfrog")
    got = b.trajectory([rs.split("gm"), rs], n_step)[0]
    assert abs(got - dh2) < 1e-13 * 24 * geo.total_volume + 1e-12 * abs(dh2)


@pytest.mark.gpu
@pytest.mark.parametrize("n_step", [1, 2, 5])
def test_steps_end_in_the_callers_links(q, n_step):
    """No copy of the links from a work buffer: that made one step slower than three separate launches."""
    gf = q.GaugeField(q.Geometry((4, 4, 4, 6)))
    gf.set_rand(q.RngState("leapfrog").split("gf"), 0.4, 1)
    gm = q.GaugeMomentum(gf.geo)
    gm.set_rand(q.RngState("leapfrog").split("gm"), 1.0)
    q.prof_reset()
    q.prof_enable(True)
    try:
        q.run_hmc_evolve_pure_gauge(gm, gf, q.GaugeAction(2.3, 0.0), None, n_step, integrator="leapfrog")
        q.synchronize()
        got = [q.prof_get(k)[1] for k in ("evolve", "force_leapfrog", "copy")]
    finally:
        q.prof_enable(False)
    assert got == [1, n_step, 0]
