"""The masked flow steps, their log-determinants and the flowed force on the
smallest lattices and on lattices whose flowed links do not fill the last
block of 32, against a plain numpy restatement."""

import numpy as np
import pytest


def dag(a):
    return np.conj(np.swapaxes(a, -1, -2))


def line(u, path):
    """Ordered product along `path` at every site (T, Z, Y, X, 4, 3, 3); mu forward, -mu - 1 backward."""
    at, out = [0] * 4, np.broadcast_to(np.eye(3, dtype=complex), u.shape[:4] + (3, 3))
    for d in path:
        mu = d if d >= 0 else -d - 1
        at[mu] -= d < 0
        m = np.roll(u[..., mu, :, :], [-at[k] for k in range(4)], [3 - k for k in range(4)])
        out = out @ (m if d >= 0 else dag(m))
        at[mu] += d >= 0
    return out


def ta(m):
    a = (m - dag(m)) / 2
    return a - np.trace(a, axis1=-2, axis2=-1)[..., None, None] / 3 * np.eye(3)


def expm(a):
    e = np.eye(a.shape[-1])
    for k in range(24, 0, -1):
        e = np.eye(a.shape[-1]) + a @ e / k
    return e


def su3_basis():
    t = np.zeros((8, 3, 3), dtype=complex)
    for a, (i, j) in ((0, (0, 1)), (3, (0, 2)), (5, (1, 2))):
        t[a, i, j] = t[a, j, i] = 1j
        t[a + 1, i, j], t[a + 1, j, i] = 1, -1
    t[2] = np.diag([1j, -1j, 0])
    t[7] = np.diag([1j, 1j, -2j]) / np.sqrt(3)
    return t


T8 = su3_basis()


def coef(m):
    return -0.5 * np.einsum("aij,...ji->...a", T8, m).real


def flow(u, steps):
    """(flowed links, sum of ln det)."""
    u, ln_det = u.copy(), 0.0
    x = np.meshgrid(*(np.arange(n) for n in u.shape[:4]), indexing="ij")
    for mask, mu, eps, size in steps:
        c = sum(line(u, [e] * size + [mu] + [-e - 1] * size)
                for nu in range(4) if nu != mu for e in (nu, -nu - 1))
        on = sum(k // size for k in x) % 2 == mask % 2
        um, cd = u[..., mu, :, :][on], dag(c)[on]
        xm = -eps * ta(um @ cd)
        n = np.swapaxes(coef(ta((T8 @ um[:, None]) @ cd[:, None])), -1, -2)
        ad = np.swapaxes(coef(xm[:, None] @ T8 - T8 @ xm[:, None]), -1, -2)
        j = np.eye(8)
        for k in range(24, 1, -1):
            j = np.eye(8) - ad @ j / k
        ln_det += np.linalg.slogdet(np.eye(8) - eps * j @ n)[1].sum()
        u[..., mu, :, :][on] = expm(xm) @ um
    return u, ln_det


def action(u, beta, steps):
    u, ln_det = flow(u, steps)
    p = sum((np.trace(line(u, [a, b, -a - 1, -b - 1]), axis1=-2, axis2=-1).real - 3).sum()
            for a in range(4) for b in range(a + 1, 4))
    return -beta / 3 * p - ln_det, u, ln_det


# extents must be multiples of 2 (size 1) or 4 (size 2): 8, 24, 240 and 128, 384 flowed links a step
CASES = [((2, 2, 2, 2), 1), ((2, 6, 2, 2), 1), ((6, 2, 4, 10), 1), ((4, 4, 4, 4), 2), ((4, 8, 4, 6), 1),
         ((12, 4, 4, 4), 2)]


@pytest.mark.gpu
@pytest.mark.parametrize("ts,size", CASES)
def test_flow_ln_det_and_force_against_numpy(q, ts, size):
    rng = np.random.default_rng(sum(ts) + size)
    shape = (*ts[::-1], 4)
    u = expm(np.einsum("...a,aij->...ij", 0.25 * rng.standard_normal((*shape, 8)), T8))
    steps = [(2, 3, 0.1, size), (1, 0, 0.07, 1), (1, 1, -0.05, size), (2, 0, 0.1, 1), (1, 3, 0.1, size)]
    fi = q.FlowInfo(q.FlowStepInfo(*s) for s in steps)
    beta = 5.5
    s0, uf, ln_det = action(u, beta, steps)
    gf = q.GaugeField(q.Geometry(ts))
    gf.from_numpy(u.reshape(-1, 4, 3, 3))
    # some hundred operations on matrices of size 1: 1e-13 is 500 units of rounding
    out, ld = q.gf_flow_and_ln_det_node(gf, fi)
    scale = np.sqrt(len(uf.reshape(-1, 9)) * 3)
    assert np.linalg.norm(np.asarray(out).ravel() - uf.ravel()) < 1e-13 * scale
    assert abs(ld - ln_det) < 1e-13 * uf.size + 1e-12 * abs(ln_det)
    assert np.array_equal(np.asarray(q.gf_flow(gf, fi)), np.asarray(out))
    back = np.asarray(q.gf_flow_inv(out, fi))
    assert np.linalg.norm(back.ravel() - u.ravel()) < 1e-12 * scale
    # the force is -1/2 of the action's gradient: five-point differences of the numpy action, h = 0.01 --
    # truncation h^4 f'''''/30 and rounding 1e-16 |S| / h, both below 1e-7 of |dS|
    ga = q.GaugeAction(beta, 0.0)
    F = q.GaugeMomentum(gf.geo)
    q.set_gm_force_flowed(F, gf, ga, fi)
    f = coef(np.asarray(F)).reshape(*shape, 8)
    w = rng.standard_normal((*shape, 8))
    w /= np.linalg.norm(w)
    X = np.einsum("...a,aij->...ij", w, T8)
    h = 0.01
    S = {k: action(expm(k * h * X) @ u, beta, steps)[0] for k in (-2, -1, 1, 2)}
    fd = (8 * (S[1] - S[-1]) - (S[2] - S[-2])) / (12 * h)
    assert abs(fd + 2 * (f * w).sum()) < 1e-7 * np.linalg.norm(2 * f)
    # and without the determinant term, through a force given on the flowed field
    pre, F2 = q.GaugeMomentum(gf.geo), q.GaugeMomentum(gf.geo)
    q.set_gm_force(pre, out, ga)
    q.set_gm_force_flowed_no_det(F2, pre, gf, fi)
    q.set_gm_force_flowed(F, gf, ga, fi, with_det=False)
    assert np.linalg.norm(np.asarray(F) - np.asarray(F2)) < 1e-14 * np.linalg.norm(np.asarray(F))


# 2 x 6 x 2 x 2 = 48 sites, 6^4 = 1296, 10^4 = 10000: the last block of 32 is half filled
@pytest.mark.gpu
@pytest.mark.parametrize("ts", [(2, 6, 2, 2), (6, 6, 6, 6), (10, 10, 10, 10)])
@pytest.mark.parametrize("n", [0, 1, 2, 5])
def test_force_leaves_no_words_beyond_its_sites(q, ts, n):
    """qnorm sums the stored field, padding sites included: it is the image's norm for every number of steps,
    whatever earlier calls left in the work buffers."""
    full = q.FlowInfo(q.FlowStepInfo(1 + i % 2, i % 4, 0.1, 1) for i in range(4))
    big = q.GaugeField(q.Geometry((8, 8, 8, 16)))
    big.set_rand(q.RngState("flowed-padding"), 0.5, 1)
    ga = q.GaugeAction(5.5, 0.0)
    q.set_gm_force_flowed(q.GaugeMomentum(big.geo), big, ga, full)
    fi = q.FlowInfo(q.FlowStepInfo(1 + i % 2, i % 4, 0.1, 1) for i in range(n))
    gf = q.GaugeField(q.Geometry(ts))
    gf.set_rand(q.RngState("flowed-padding"), 0.3, 1)
    pre, F, F2 = (q.GaugeMomentum(gf.geo) for _ in range(3))
    q.set_gm_force_flowed(F, gf, ga, fi, with_det=False)
    q.set_gm_force(pre, q.gf_flow(gf, fi), ga)
    q.set_gm_force_flowed_no_det(F2, pre, gf, fi)
    for f in (F, F2):
        image = float((np.abs(np.asarray(f)) ** 2).sum())
        assert abs(f.qnorm() - image) < 1e-12 * image  # two orders of one sum of positive terms
    assert np.linalg.norm(np.asarray(F) - np.asarray(F2)) < 1e-14 * np.linalg.norm(np.asarray(F))


@pytest.mark.gpu
def test_inverse_flow_at_many_links(q):
    """The inverse on more links than a block per SM holds (16^4: 32768 a step, and 12 x 10 x 10 x 14: 8400, no
    multiple of 32): the iterations run on all of the GPU.  2048 links are 64 warps of one chain of iterations
    each; 16 times as many, 7 warps an SM, take 1.7 times as long (with one warp of a block at work and seven waiting,
    6.6 times)."""
    import time
    fi = q.FlowInfo(q.FlowStepInfo(1 + i % 2, i % 4, 0.1, 1) for i in range(8))
    t = []
    for ts in [(8, 8, 8, 8), (12, 10, 10, 14), (16, 16, 16, 16)]:
        gf = q.GaugeField(q.Geometry(ts))
        gf.set_rand(q.RngState("inverse"), 0.3, 1)
        out = q.gf_flow(gf, fi)
        back = q.gf_flow_inv(out, fi)
        a, b = np.asarray(gf), np.asarray(back)
        assert np.linalg.norm(a - b) < 1e-12 * np.linalg.norm(a)
        best = 1e9
        for _ in range(5):
            q.synchronize()
            t0 = time.perf_counter()
            q.gf_flow_inv(back, out, fi)
            q.synchronize()
            best = min(best, time.perf_counter() - t0)
        t.append(best)
    assert t[2] < 4 * t[0], t
