"""The flow adjoint with every step's stage fields kept, against the same
gradient through recomputed segments (a flow too long to keep), and the
release of what it keeps."""

import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("c1", [0.0, -0.331])
@pytest.mark.parametrize("single", [False, True])
def test_kept_and_recomputed_gradients_agree(q, c1, single):
    ts, eps, steps = (4, 4, 4, 6), 0.01, 5
    gf = q.GaugeField(q.Geometry(ts))
    gf.set_rand(q.RngState("adjoint-kept"), 0.3, 1)
    g = gf.copy(precision=q.F32 if single else q.F64)
    # all five steps at once (kept), the loss's gradient pulled back step by step: five vjp calls of one step
    loss, grad = q.gf_flow_action_grad(g, eps, steps, 5.5, c1=c1, checkpoint_every=2)
    again = q.gf_flow_action_grad(g, eps, steps, 5.5, c1=c1, checkpoint_every=2)
    assert again[0] == loss and np.array_equal(np.asarray(again[1]), np.asarray(grad))
    w = [g.copy()]
    for _ in range(steps):
        w.append(w[-1].copy())
        q.gf_wilson_flow_step(w[-1], eps, c1=c1)
    lam = q.GaugeMomentum(gf.geo, precision=g.precision)
    q.set_gm_force(lam, w[-1], q.GaugeAction(5.5, 0.0))
    lam *= -2.0
    for u in reversed(w[:-1]):
        lam = q.gf_wilson_flow_vjp(u, eps, 1, lam, c1=c1)
    tol = 500 * (6e-8 if single else 1.1e-16)
    assert np.linalg.norm(np.asarray(lam) - np.asarray(grad)) < tol * np.linalg.norm(np.asarray(grad))
    v = q.gf_wilson_flow_vjp(g, eps, steps, np_field(q, gf, w[-1]), c1=c1, checkpoint_every=3)
    assert np.linalg.norm(np.asarray(v) - np.asarray(grad)) < tol * np.linalg.norm(np.asarray(grad))


def np_field(q, gf, flowed):
    lam = q.GaugeMomentum(gf.geo, precision=flowed.precision)
    q.set_gm_force(lam, flowed, q.GaugeAction(5.5, 0.0))
    lam *= -2.0
    return lam


@pytest.mark.gpu
def test_kept_fields_are_given_back(q):
    gf = q.GaugeField(q.Geometry((8, 8, 8, 8)))
    gf.set_rand(q.RngState("adjoint-kept"), 0.3, 1)
    loss, grad = q.gf_flow_action_grad(gf, 0.02, 10, 5.5)
    first = np.asarray(grad)
    field = 4 * 8 ** 4 * 144
    assert q.release_field_pool() >= 60 * field  # ten steps' links and five stage fields each
    loss2, grad2 = q.gf_flow_action_grad(gf, 0.02, 10, 5.5)
    assert loss2 == loss and np.array_equal(np.asarray(grad2), first)
    # a flow whose stage fields exceed the bound recomputes its segments: 1900 steps of 2.4 MB fields
    long = q.gf_flow_action_grad(gf, 1e-5, 1900, 5.5, checkpoint_every=64)
    short = q.gf_flow_action_grad(gf, 1e-5 * 95, 20, 5.5)
    assert abs(long[0] - short[0]) < 1e-6 * abs(short[0])  # the flow times agree, the step errors are eps^3
    a, b = np.asarray(long[1]), np.asarray(short[1])
    assert np.linalg.norm(a - b) < 1e-6 * np.linalg.norm(b)
    q.release_field_pool()


@pytest.mark.gpu
def test_many_checkpoints_have_buffers_of_their_own(q):
    """A flow of 1900 steps (26 GB of links and stage fields of 8^4, not kept) with 950 checkpoints, and with 30:
    the same launches on the same links, so the same bits."""
    gf = q.GaugeField(q.Geometry((8, 8, 8, 8)))
    gf.set_rand(q.RngState("adjoint-kept"), 0.3, 1)
    few = q.gf_flow_action_grad(gf, 1e-4, 1900, 5.5, checkpoint_every=64)
    many = q.gf_flow_action_grad(gf, 1e-4, 1900, 5.5, checkpoint_every=2)
    assert many[0] == few[0] and np.array_equal(np.asarray(many[1]), np.asarray(few[1]))
    lam = np_field(q, gf, gf)
    few, many = (q.gf_wilson_flow_vjp(gf, 1e-4, 1900, lam, checkpoint_every=e) for e in (64, 2))
    assert np.array_equal(np.asarray(many), np.asarray(few))
    q.release_field_pool()
