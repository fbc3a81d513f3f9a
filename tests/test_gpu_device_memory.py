"""A device that another program has filled: what the library does when an
allocation of its own fails.  Each case is a process of its own, so that the
library starts without buffers of earlier tests."""

import os
import subprocess
import sys
import textwrap

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PRELUDE = '''
import numpy as np, torch
import qlat_b200 as q

def links(ts):
    gf = q.GaugeField(q.Geometry(ts))
    gf.set_rand(q.RngState("memory"), 0.3, 1)
    return gf

class Filled:
    """All of the device but `spare` bytes in other hands."""
    def __init__(self, spare):
        self.spare = spare
    def __enter__(self):
        q.synchronize()
        torch.cuda.empty_cache()
        self.t = torch.empty(torch.cuda.mem_get_info()[0] - self.spare, dtype=torch.uint8, device="cuda")
    def __exit__(self, *a):
        del self.t
        torch.cuda.empty_cache()
'''


def run(q, code):
    r = subprocess.run([sys.executable, "-c", PRELUDE + textwrap.dedent(code)], cwd=ROOT, capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-4000:]


@pytest.mark.gpu
def test_transfer_without_room_leaves_the_next_ones_usable(q):
    """The staging buffer has 2 MB, a transfer of 75 MB cannot enlarge it, and the next needs the 2 MB again."""
    run(q, '''
        a, b = links((8, 8, 8, 8)), links((16, 16, 16, 32))
        small = a.to_numpy()
        with Filled(32 << 20):
            for _ in range(2):
                try:
                    b.to_numpy()
                except q.QlatB200Error:
                    pass
                else:
                    raise SystemExit("the transfer found room")
                assert np.array_equal(a.to_numpy(), small)
                a.from_numpy(small)
                assert abs(q.gf_avg_plaq(a)) < 1
        big = b.to_numpy()
        b.from_numpy(big)
        assert np.array_equal(b.to_numpy(), big) and np.array_equal(a.to_numpy(), small)
    ''')


@pytest.mark.gpu
def test_idle_memory_is_given_up_for_every_kind_of_buffer(q):
    """The flow adjoint holds 9 GB for its next call and the device has 64 MB left: staging, work fields of a trajectory,
    the work pool, fields, and batches find room all the same, each with the buffers held anew."""
    run(q, '''
        g, big = links((16, 16, 16, 16)), links((16, 16, 16, 32))
        gm, F = q.GaugeMomentum(big.geo), q.GaugeMomentum(big.geo)
        gm.set_rand(q.RngState("memory"), 1.0)
        ga, fi = q.GaugeAction(5.5, 0.0), q.FlowInfo([q.FlowStepInfo(1, 0, 0.1, 1)])
        want = q.gf_flow_action_grad(g, 0.01, 40, 5.5)
        made = []
        for use in (lambda: q.run_hmc_evolve_pure_gauge(gm, big, ga, None, 1, 0.1, integrator="leapfrog"),
                    lambda: q.set_gm_force_flowed(F, big, ga, fi),
                    lambda: made.append(q.ChainBatch([(8, 8, 8, 8)] * 64, [5.5] * 64)),
                    lambda: made.append(big.copy()),
                    lambda: big.to_numpy()):
            q.gf_flow_action_grad(g, 0.01, 40, 5.5)
            with Filled(64 << 20):
                use()
                assert torch.cuda.mem_get_info()[0] > 7 << 30  # what the adjoint held and the call did not take
        # a short device cannot take the fields of a running gradient from it
        with Filled(3 << 30):
            loss, grad = q.gf_flow_action_grad(g, 0.01, 40, 5.5)
        assert loss == want[0] and np.array_equal(np.asarray(grad), np.asarray(want[1]))
        # and the work pool is given back too
        assert q.release_field_pool() > 0 and q.release_field_pool() == 0
    ''')


@pytest.mark.gpu
def test_improved_charge_needs_no_room(q):
    """The five loops' terms with and without room for the field of lines (1.2 KB a site in FP64): the same products
    in the same order.  Extents of 1 to 3 (lines that wrap around) and partly filled blocks of 64 sites."""
    run(q, '''
        from qlat_b200._lib import call
        for ts in ((16, 16, 16, 32), (1, 2, 3, 20000), (17, 15, 19, 20)):
            for precision in (q.F64, q.F32):
                gf = links(ts).copy(precision=precision)
                topf = q.FieldRealD(gf.geo, 5, precision=precision)
                out = []
                for spare in (None, 24 << 20):  # (the lines are 55 to 151 MB)
                    q.release_field_pool()
                    n0 = q.launch_count()
                    if spare is None:
                        out.append(q.gf_topology_terms(gf))
                    else:
                        with Filled(spare):
                            out.append(q.gf_topology_terms(gf))
                            call("qgb_clf_topology_field_5_terms", topf.handle, gf.handle)
                    out.append(q.launch_count() - n0)
                assert out[1] == 3 and out[3] == 4, "three kernels with the lines, two without"
                assert np.array_equal(out[0], out[2]), (ts, precision, out)
                assert np.array_equal(np.asarray(topf), np.asarray(q.gf_topology_terms_field(gf)))
    ''')


@pytest.mark.gpu
def test_pairs_of_sites_without_room_run_in_the_scalar_form(q):
    """Three packed fields of 47 MB and 64 MB of room: the first one fits, is given back, and trajectory and flow run as
    on a lattice that cannot be paired; with room again they run in pairs."""
    run(q, '''
        gf = links((16, 16, 16, 32))
        gm = q.GaugeMomentum(gf.geo)
        gm.set_rand(q.RngState("memory"), 1.0)
        ga, u, p = q.GaugeAction(2.13, -0.331), gf.copy(), gm.copy()
        g32 = gf.copy(precision=q.F32)

        def packed(f):
            q.prof_reset()
            q.prof_enable(True)
            f()
            q.synchronize()
            q.prof_enable(False)
            return q.prof_get("pair_pack")[1]

        def trajectory():
            u.__imatmul__(gf)
            p.__imatmul__(gm)
            q.run_hmc_evolve_pure_gauge(p, u, ga, None, 8, precision="mixed")

        def flow():
            g32.__imatmul__(gf)
            q.gf_wilson_flow_step(g32, 0.02, c1=-0.331)

        old = q.force_get_variant(q.F32, True)
        q.force_set_variant(q.F32, True, 10)
        trajectory(), flow()  # the scalar form, and the work fields that it needs
        want = np.asarray(u), np.asarray(g32)
        q.force_set_variant(q.F32, True, old)
        q.release_field_pool()
        with Filled(64 << 20):
            free = torch.cuda.mem_get_info()[0]
            assert packed(trajectory) == 0 and packed(flow) == 0
            assert torch.cuda.mem_get_info()[0] == free
            trajectory(), trajectory()  # recorded and replayed
            got = [(np.asarray(u), np.asarray(g32))]
        assert packed(trajectory) == 4 and packed(flow) == 2
        trajectory(), trajectory()
        got.append((np.asarray(u), np.asarray(g32)))
        for links_, flowed in got:  # FP32: the tolerance of the paired form's own tests
            assert np.abs(links_ - want[0]).max() < 2e-5 and np.abs(flowed - want[1]).max() < 2e-5
    ''')
