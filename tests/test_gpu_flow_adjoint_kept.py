"""The flow adjoint with every step's links and stage fields kept, with those
of a recomputed segment kept, and with every step recomputed: the same
gradient.  The bounds on what it keeps, over all lattices; what it does when
the device is short of memory; and the release of what it keeps."""

import numpy as np
import pytest


@pytest.fixture
def memory(q):
    """set_flow_adjoint_memory, with the defaults and an empty pool before and after."""
    q.set_flow_adjoint_memory()
    q.release_field_pool()
    yield q.set_flow_adjoint_memory
    q.set_flow_adjoint_memory()
    q.release_field_pool()


def links(q, ts, single=False):
    gf = q.GaugeField(q.Geometry(ts))
    gf.set_rand(q.RngState("adjoint-kept"), 0.3, 1)
    return gf.copy(precision=q.F32) if single else gf


def force_at(q, flowed):
    lam = q.GaugeMomentum(flowed.geo, precision=flowed.precision)
    q.set_gm_force(lam, flowed, q.GaugeAction(5.5, 0.0))
    lam *= -2.0
    return lam


def launches(q, f):
    """(flow stages, pulled-back steps) that f() launches."""
    q.prof_reset()
    q.prof_enable(True)
    try:
        f()
        q.synchronize()
        return q.prof_get("flow_stage")[1], q.prof_get("flow_adjoint")[1]
    finally:
        q.prof_enable(False)


MODES = [(1 << 40, 1 << 40), (0, 1 << 40), (0, 0)]  # flow kept, segments kept, nothing kept


@pytest.mark.gpu
@pytest.mark.parametrize("c1", [0.0, -0.331])
@pytest.mark.parametrize("single", [False, True])
@pytest.mark.parametrize("every", [1, 3, 4, 100])
def test_kept_and_recomputed_gradients_agree(q, memory, c1, single, every):
    ts, eps, steps = (4, 4, 4, 6), 0.01, 7
    g = links(q, ts, single)
    # the loss's gradient pulled back step by step: seven vjp calls of one step
    w = [g.copy()]
    for _ in range(steps):
        w.append(w[-1].copy())
        q.gf_wilson_flow_step(w[-1], eps, c1=c1)
    top = force_at(q, w[-1])
    lam = top.copy()
    for u in reversed(w[:-1]):
        lam = q.gf_wilson_flow_vjp(u, eps, 1, lam, c1=c1)
    lam = np.asarray(lam)
    got = []
    for flow, segment in MODES:
        memory(flow, segment)
        for _ in range(2):  # the buffers new, then held
            loss, grad = q.gf_flow_action_grad(g, eps, steps, 5.5, c1=c1, checkpoint_every=every)
            vjp = q.gf_wilson_flow_vjp(g, eps, steps, top, c1=c1, checkpoint_every=every)
            got.append((loss, np.asarray(grad), np.asarray(vjp)))
    # the same stages on the same links
    for loss, grad, vjp in got[1:]:
        assert loss == got[0][0] and np.array_equal(grad, got[0][1]) and np.array_equal(vjp, got[0][2])
    tol = 500 * (6e-8 if single else 1.1e-16)
    for m in got[0][1:]:
        assert np.linalg.norm(m - lam) < tol * np.linalg.norm(lam)


@pytest.mark.gpu
def test_each_mode_runs(q, memory):
    """7 steps, checkpoints every 3: segments of 3, 3 and 1 steps."""
    g = links(q, (4, 4, 4, 4))
    lam = force_at(q, g)
    grad = lambda: q.gf_flow_action_grad(g, 0.01, 7, 5.5, checkpoint_every=3)  # noqa: E731
    vjp = lambda: q.gf_wilson_flow_vjp(g, 0.01, 7, lam, checkpoint_every=3)  # noqa: E731
    # stages: the flow; the segments again; or the steps but each segment's last, then every step once more
    for (flow, segment), again, to_checkpoints in zip(MODES, (0, 21, 12 + 21), (21, 18, 18)):
        memory(flow, segment)
        assert launches(q, grad) == (21 + again, 7)
        assert launches(q, vjp) == (to_checkpoints + again, 7)


@pytest.mark.gpu
def test_kept_fields_are_given_back(q, memory):
    gf = links(q, (8, 8, 8, 8))
    loss, grad = q.gf_flow_action_grad(gf, 0.02, 10, 5.5)
    first = np.asarray(grad)
    field = 4 * 8 ** 4 * 144
    assert q.release_field_pool() == 60 * field  # ten steps' links and five stage fields each
    loss2, grad2 = q.gf_flow_action_grad(gf, 0.02, 10, 5.5)
    assert loss2 == loss and np.array_equal(np.asarray(grad2), first)
    # a flow whose stage fields exceed the bound recomputes its segments: 1900 steps of 2.4 MB fields
    long = q.gf_flow_action_grad(gf, 1e-5, 1900, 5.5, checkpoint_every=64)
    short = q.gf_flow_action_grad(gf, 1e-5 * 95, 20, 5.5)
    assert abs(long[0] - short[0]) < 1e-6 * abs(short[0])  # the flow times agree, the step errors are eps^3
    a, b = np.asarray(long[1]), np.asarray(short[1])
    assert np.linalg.norm(a - b) < 1e-6 * np.linalg.norm(b)


@pytest.mark.gpu
def test_bound_counts_six_fields_a_step_of_all_lattices(q, memory):
    a, b = links(q, (8, 8, 8, 8)), links(q, (8, 8, 8, 4))
    fa, fb = 4 * 8 ** 4 * 144, 2 * 8 ** 4 * 144
    grad = lambda g, steps: q.gf_flow_action_grad(g, 0.01, steps, 5.5, checkpoint_every=2)  # noqa: E731
    keep = []  # (momenta alive: none of them goes to the field pool)
    memory(60 * fa, 0)
    assert launches(q, lambda: keep.append(grad(a, 10)))[0] == 30  # kept: 60 fields
    assert launches(q, lambda: keep.append(grad(a, 11)))[0] > 33  # 66 fields are too many
    assert q.release_field_pool() == 8 * fa  # 6 checkpoints and a segment's 2 links: less than the 60 fields went with them
    keep += [grad(a, 10), grad(b, 10)]  # 60 fields and 60 half ones: not both
    assert q.release_field_pool() == 60 * fb
    keep += [grad(a, 5), grad(b, 10)]
    assert q.release_field_pool() == 30 * fa + 60 * fb


@pytest.mark.gpu
def test_many_checkpoints_have_buffers_of_their_own(q, memory):
    """A flow of 1900 steps (26 GB of links and stage fields of 8^4, not kept) with 950 checkpoints, and with 30:
    the same launches on the same links, so the same bits."""
    gf = links(q, (8, 8, 8, 8))
    few = q.gf_flow_action_grad(gf, 1e-4, 1900, 5.5, checkpoint_every=64)
    many = q.gf_flow_action_grad(gf, 1e-4, 1900, 5.5, checkpoint_every=2)
    assert many[0] == few[0] and np.array_equal(np.asarray(many[1]), np.asarray(few[1]))
    lam = force_at(q, gf)
    few, many = (q.gf_wilson_flow_vjp(gf, 1e-4, 1900, lam, checkpoint_every=e) for e in (64, 2))
    assert np.array_equal(np.asarray(many), np.asarray(few))


@pytest.mark.gpu
@pytest.mark.parametrize("spare_fields", [120, 40])
def test_short_of_device_memory(q, memory, spare_fields):
    """A 16^4 flow of 20 steps (120 fields of 37.7 MB) beside another program that leaves the device less than that:
    the steps are recomputed, with a segment's 40 stage fields or without, and the gradient is the same."""
    import torch
    g = links(q, (16, 16, 16, 16))
    grad = lambda: q.gf_flow_action_grad(g, 0.01, 20, 5.5, checkpoint_every=8)  # noqa: E731
    want = grad()  # (and the work fields are there)
    q.release_field_pool()
    q.synchronize()
    torch.cuda.empty_cache()
    field = 4 * 16 ** 4 * 144
    other = torch.empty(torch.cuda.mem_get_info()[0] - spare_fields * field, dtype=torch.uint8, device="cuda")
    try:
        out = []
        stages = launches(q, lambda: out.append(grad()))[0]
    finally:
        del other
        torch.cuda.empty_cache()
    assert stages > 60
    assert out[0][0] == want[0] and np.array_equal(np.asarray(out[0][1]), np.asarray(want[1]))
