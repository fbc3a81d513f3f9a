"""The clover and improved-charge kernels where their tiling can go wrong:
extents of 1 to 3 (the larger loops wrap), site counts around the 64 sites of
a block, and the z-slab sweep of large time slices, against the oracle."""

import numpy as np
import pytest

SHAPES = [(1, 2, 3, 5), (2, 2, 2, 2), (3, 3, 3, 3), (4, 4, 4, 1), (13, 5, 1, 1), (5, 7, 3, 4), (16, 16, 96, 2)]


@pytest.mark.gpu
@pytest.mark.parametrize("ts", SHAPES)
@pytest.mark.parametrize("single", [False, True])
def test_clover_and_improved_charge(q, oracle, ts, single):
    rs, ro = q.RngState("clover-shapes"), oracle.RngState("clover-shapes")
    gf = q.GaugeField(q.Geometry(ts))
    gf.set_rand(rs, 0.3, 1)
    ref = np.ascontiguousarray(np.asarray(gf))
    if single:
        gf = gf.copy(precision=q.F32)
        ref = np.ascontiguousarray(np.asarray(gf))
    # per site: sums of some 100 products of matrices of size 1, FP64 1e-16 each and FP32 6e-8
    tol = 3e-5 if single else 5e-14
    e_ref, q_ref = oracle.gf_energy_density_field(ref, ts), oracle.clf_topology_field(ref, ts)
    e = np.asarray(q.gf_energy_density_field(gf))[:, 0]
    c = np.asarray(q.gf_topology_field_clf(gf))[:, 0]
    assert np.abs(e - e_ref).max() <= tol * np.abs(e_ref).max()
    assert np.abs(c - q_ref).max() <= tol * max(np.abs(q_ref).max(), np.abs(e_ref).max() / 40)
    assert abs(q.gf_energy_density(gf) - e_ref.mean()) <= tol * e_ref.mean()
    assert abs(q.gf_topology_clf(gf) - q_ref.sum()) <= tol * np.abs(q_ref).sum() + 1e-15
    if len(ref) > 1000:
        return  # the oracle walks the larger loops link by link
    t_ref = oracle.clf_topology_field_5_terms(ref, ts)
    scale = np.abs(t_ref).max(axis=0) + np.abs(e_ref).max() / 40
    t = np.asarray(q.gf_topology_terms_field(gf))
    assert (np.abs(t - t_ref).max(axis=0) <= tol * scale).all()
    assert np.abs(np.asarray(q.gf_topology_field(gf))[:, 0] - t_ref.sum(axis=1)).max() <= tol * scale.sum()
    assert np.abs(q.gf_topology_terms(gf) - t_ref.sum(axis=0)).max() <= tol * scale.max() * len(ref)
