"""The work that users of this framework have it do, as cases to time and compare.

A case is a dict of plain values: its "kind" names the path and the rest its
sizes and options.  `prepare` makes what a program holds before the call (the
fields, filled from a seed), `run` is one pass through the public API, and
`exact` the same numbers in 64 bits from plain torch.

Kinds:
  hmc       one trajectory of run_hmc_pure_gauge from a given configuration
  force     set_gm_force
  flow      gf_wilson_flow of a copy of the configuration, then its clover-charge density
  measure   plaquette, energy-density field and clover-charge field
  topology  the five terms of the 5-loop improved charge density
  adjoint   gradient of the flowed action by the flow adjoint
  flowed    force of flowed HMC (masked flows and their log-determinants)
  batch     proposals of many independent chains at once

Links are independent random SU(3) matrices near the unit matrix, with the
plaquettes that production couplings have.  Trajectories start from a copy of
the same configuration in every pass, so passes are alike.
"""

import math

import numpy as np
import torch
from torch.utils.checkpoint import checkpoint

import qlat_b200 as q

IWASAKI, DBW2 = -0.331, -1.4008


def listed():
    return [
        # production HMC: the README's and the benchmark's workload
        {"name": "hmc-mixed-24x64", "kind": "hmc", "x": 24, "y": 24, "z": 24, "t": 64, "beta": 2.13, "c1": IWASAKI,
         "integrator": "force-gradient", "steps": 8, "precision": "mixed"},
        # the API's defaults (FP64, force-gradient, 6 steps) on a common middle size
        {"name": "hmc-fp64-16x32", "kind": "hmc", "x": 16, "y": 16, "z": 16, "t": 32, "beta": 2.13, "c1": IWASAKI,
         "integrator": "force-gradient", "steps": 6, "precision": "fp64"},
        # the benchmark's small chain, where launches and latency count
        {"name": "hmc-fp64-8", "kind": "hmc", "x": 8, "y": 8, "z": 8, "t": 8, "beta": 5.5, "c1": 0.0,
         "integrator": "leapfrog", "steps": 6, "precision": "fp64"},
        # ragged extents (partly filled blocks of sites) with the third action
        {"name": "hmc-mixed-odd", "kind": "hmc", "x": 11, "y": 10, "z": 13, "t": 18, "beta": 0.87, "c1": DBW2,
         "integrator": "leapfrog", "steps": 10, "precision": "mixed"},
        # a force by itself: integrators that users write in Python (Qlattice's example drivers) call it
        {"name": "force-fp64-24x64", "kind": "force", "x": 24, "y": 24, "z": 24, "t": 64, "beta": 2.13, "c1": IWASAKI},
        # scale setting: the benchmark's 32^4 Wilson flow with t^2 E after each step
        {"name": "flow-fp64-32", "kind": "flow", "x": 32, "y": 32, "z": 32, "t": 32, "c1": 0.0, "eps": 0.05,
         "steps": 4, "precision": "fp64"},
        # the same with FP32 links and the Iwasaki flow, on a shape that is not a cube
        {"name": "flow-fp32-24x48", "kind": "flow", "x": 24, "y": 24, "z": 24, "t": 48, "c1": IWASAKI, "eps": 0.02,
         "steps": 4, "precision": "fp32"},
        # densities of one stored configuration
        {"name": "measure-fp64-24x48", "kind": "measure", "x": 24, "y": 24, "z": 24, "t": 48, "precision": "fp64"},
        # topology measurement of a stored configuration
        {"name": "topology-fp64-16x32", "kind": "topology", "x": 16, "y": 16, "z": 16, "t": 32, "precision": "fp64"},
        # the benchmark's flow adjoint: backward through 40 steps
        {"name": "adjoint-16", "kind": "adjoint", "x": 16, "y": 16, "z": 16, "t": 16, "beta": 5.8, "eps": 0.05,
         "steps": 40},
        # flowed HMC: one force through a full set of 16 masked steps
        {"name": "flowed-8x16", "kind": "flowed", "x": 8, "y": 8, "z": 8, "t": 16, "beta": 2.13, "c1": IWASAKI,
         "eps": 0.1, "eps2": -0.01},
        # the benchmark's 256 chains on four sizes
        {"name": "batch-mixed-256", "kind": "batch", "chains": 256, "extents": "4,6,8,12", "steps": 10,
         "precision": "mixed"},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _extents(rng, v_max, step=1):
    """A lattice of at most v_max sites: spatial extents near one another, a longer time extent as often as not."""
    while True:
        v = math.exp(rng.uniform(math.log(600), math.log(v_max)))
        aspect = rng.choice([1, 1, 2, 2.67])
        side = (v / aspect) ** 0.25
        e = [max(4, step * int(round(side * rng.uniform(0.85, 1.15) / step))) for _ in range(3)]
        e.append(max(4, step * int(round(aspect * side * rng.uniform(0.9, 1.1) / step))))
        if e[0] * e[1] * e[2] * e[3] <= v_max:
            return dict(zip("xyzt", e))


def draw(rng):
    kind = rng.choice(["hmc", "hmc", "hmc", "force", "flow", "flow", "measure", "topology", "adjoint", "flowed", "batch"])
    beta, c1 = rng.choice([(5.5, 0.0), (6.0, 0.0), (2.13, IWASAKI), (2.6, IWASAKI), (0.87, DBW2)])
    precision = rng.choice(["fp64", "low"])
    if kind == "hmc":
        integrator = rng.choice(["force-gradient", "leapfrog"])
        steps = rng.randint(4, 8) if integrator == "force-gradient" else rng.randint(5, 12)
        return {"kind": kind, **_extents(rng, 800000 if precision == "low" else 250000), "beta": beta, "c1": c1,
                "integrator": integrator, "steps": steps, "precision": "fp64" if precision == "fp64" else "mixed"}
    if kind == "force":
        return {"kind": kind, **_extents(rng, 800000), "beta": beta, "c1": c1}
    if kind == "flow":
        return {"kind": kind, **_extents(rng, 700000), "c1": c1, "eps": {0.0: 0.05, IWASAKI: 0.02, DBW2: 0.005}[c1],
                "steps": rng.randint(1, 6), "precision": "fp64" if precision == "fp64" else "fp32"}
    if kind in ("measure", "topology"):
        return {"kind": kind, **_extents(rng, 600000 if kind == "measure" else 200000),
                "precision": "fp64" if precision == "fp64" else "fp32"}
    if kind == "adjoint":
        return {"kind": kind, **_extents(rng, 50000), "beta": 5.8, "eps": rng.choice([0.02, 0.05]),
                "steps": rng.randint(4, 40)}
    if kind == "flowed":
        two = rng.random() < 0.5
        return {"kind": kind, **_extents(rng, 8000, 4), "beta": beta, "c1": c1, "eps": 0.1, "eps2": -0.01 if two else 0.0}
    sides = sorted(rng.sample([4, 5, 6, 7, 8, 10, 12], rng.randint(2, 4)))
    return {"kind": "batch", "chains": _log_uniform(rng, 8, 200), "extents": ",".join(map(str, sides)),
            "steps": rng.randint(5, 10), "precision": "fp64" if precision == "fp64" else "mixed"}


# ---------------------------------------------------------------------------
# inputs

def _site(case):
    return (case["x"], case["y"], case["z"], case["t"])


def _volume(case):
    if case["kind"] == "batch":
        return sum(s ** 4 for s in _chain_sides(case))
    return case["x"] * case["y"] * case["z"] * case["t"]


def _chain_sides(case):
    sides = [int(s) for s in case["extents"].split(",")]
    return [sides[c * len(sides) // case["chains"]] for c in range(case["chains"])]


def _chain_betas(case):
    return [float(b) for b in np.linspace(5.6, 6.2, case["chains"])]


def _su3(basis):
    """sum_a basis[..., a] T_a, T_a the su(3) basis with tr T_a T_b = -2 delta_ab."""
    b = basis.unbind(-1)
    s3, o = b[7] / math.sqrt(3.0), torch.zeros_like(b[0])
    re = torch.stack([o, b[1], b[4], -b[1], o, b[6], -b[4], -b[6], o], -1)
    im = torch.stack([b[2] + s3, b[0], b[3], b[0], s3 - b[2], b[5], b[3], b[5], -2 * s3], -1)
    return torch.complex(re, im).unflatten(-1, (3, 3))


def _mm(a, b):
    return sum(a[..., :, k:k + 1] * b[..., k:k + 1, :] for k in range(3))


def _dag(a):
    return a.transpose(-1, -2).conj()


def _exp(a):
    one = torch.eye(3, dtype=a.dtype, device=a.device)
    e = a / 20 + one
    for n in range(19, 0, -1):
        e = _mm(a, e) / n + one
    return e


def _links(sites, seed, sigma=0.3, stream=0):
    """Random links in the reference image: (sites, 4, 3, 3), complex128."""
    g = torch.Generator(device="cuda").manual_seed(1000003 * int(seed) + stream)
    basis = torch.randn((sites, 4, 8), dtype=torch.float64, device="cuda", generator=g)
    return _exp(_su3(basis * (sigma / math.sqrt(2.0)))).contiguous()


def _gauge_field(case, seed, precision=q.F64):
    u = _links(_volume(case), seed)
    torch.cuda.synchronize()
    gf = q.GaugeField(q.Geometry(_site(case)), precision=precision)
    gf.upload_device(u.data_ptr())
    q.synchronize()
    return gf


def _buffer(case, *shape, dtype=torch.complex128):
    return torch.empty((_volume(case), *shape), dtype=dtype, device="cuda")


def _flow_info(case):
    fi = q.FlowInfo()
    for mask, mu, eps, size in _flow_steps(case):
        fi.add_flow(mask, mu, eps, size)
    return fi


def _flow_steps(case):
    out = []
    for mu in (3, 2, 1, 0):
        for size, eps in ((1, case["eps"]), (2, case["eps2"])):
            if eps != 0.0:
                out += [(2, mu, eps, size), (1, mu, eps, size)]
    return out


def _prec(case):
    return q.F32 if case["precision"] == "fp32" else q.F64


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case, "kind": kind}
    if kind == "batch":
        sides = _chain_sides(case)
        b = q.ChainBatch([(n,) * 4 for n in sides], _chain_betas(case))
        u = _links(_volume(case), seed).cpu().numpy()
        at = 0
        for c, n in enumerate(sides):
            b.chain_from_numpy(c, u[at:at + n ** 4])
            at += n ** 4
        s["batch"] = b
        s["rs"] = [q.RngState(f"batch-{seed}").split(f"chain-{c}") for c in range(len(sides))]
        return s
    s["start"] = _gauge_field(case, seed, _prec(case) if "precision" in case else q.F64)
    if kind == "hmc":
        s["ga"] = q.GaugeAction(case["beta"], case["c1"])
        s["rs"] = q.RngState(f"hmc-{seed}")
        s["gf"] = q.GaugeField(q.Geometry(_site(case)))
        s["links"] = _buffer(case, 4, 3, 3)
    elif kind in ("force", "flowed"):
        s["ga"] = q.GaugeAction(case["beta"], case["c1"])
        s["gm"] = q.GaugeMomentum(q.Geometry(_site(case)))
        s["force"] = _buffer(case, 4, 3, 3)
        if kind == "flowed":
            s["fi"] = _flow_info(case)
    elif kind == "flow":
        s["gf"] = q.GaugeField(q.Geometry(_site(case)), precision=_prec(case))
        s["c"], s["links"] = _buffer(case, 1, dtype=torch.float64), _buffer(case, 4, 3, 3)
    elif kind == "measure":
        s["e"], s["c"] = _buffer(case, 1, dtype=torch.float64), _buffer(case, 1, dtype=torch.float64)
    elif kind == "topology":
        s["terms"] = _buffer(case, 5, dtype=torch.float64)
    elif kind == "adjoint":
        s["grad"] = _buffer(case, 4, 3, 3)
    return s


# ---------------------------------------------------------------------------
# one pass

def run(s):
    case, kind = s["case"], s["kind"]
    if kind == "hmc":
        s["gf"] @= s["start"]
        flag, delta_h = q.run_hmc_pure_gauge(s["gf"], s["ga"], 1, s["rs"], n_step=case["steps"],
                                             integrator=case["integrator"], precision=case["precision"],
                                             is_always_accept=True)
        s["gf"].download_device(s["links"].data_ptr())
        return {"accepted": bool(flag), "delta_h": np.array([delta_h]), "links": s["links"]}
    if kind == "force":
        q.set_gm_force(s["gm"], s["start"], s["ga"])
        s["gm"].download_device(s["force"].data_ptr())
        return s["force"]
    if kind == "flow":
        s["gf"] @= s["start"]
        e = q.gf_wilson_flow(s["gf"], case["eps"] * case["steps"], case["steps"], c1=case["c1"])
        q.gf_topology_field_clf(s["gf"]).download_device(s["c"].data_ptr())
        s["gf"].download_device(s["links"].data_ptr())
        return {"energy": np.array(e), "charge": s["c"], "links": s["links"]}
    if kind == "measure":
        plaq = q.gf_avg_plaq(s["start"])
        q.gf_energy_density_field(s["start"]).download_device(s["e"].data_ptr())
        q.gf_topology_field_clf(s["start"]).download_device(s["c"].data_ptr())
        return {"plaq": np.array([plaq]), "energy": s["e"], "charge": s["c"]}
    if kind == "topology":
        q.gf_topology_terms_field(s["start"]).download_device(s["terms"].data_ptr())
        return s["terms"]
    if kind == "adjoint":
        loss, grad = q.gf_flow_action_grad(s["start"], case["eps"], case["steps"], case["beta"])
        grad.download_device(s["grad"].data_ptr())
        return {"loss": np.array([loss]), "grad": s["grad"]}
    if kind == "flowed":
        q.set_gm_force_flowed(s["gm"], s["start"], s["ga"], s["fi"])
        s["gm"].download_device(s["force"].data_ptr())
        return s["force"]
    # batch: proposals only, so the chains stay where they are
    dh = s["batch"].trajectory(s["rs"], case["steps"], precision=case["precision"])
    return {"delta_h": dh, "plaq": s["batch"].plaq()}


# ---------------------------------------------------------------------------
# what a pass cannot do without

MUL = 198.0  # flops of a 3x3 complex product


def _force_flops(c1):
    """Per link.  The two-link products of a site shared by the links that read them: 3 + 6 products for the
    plaquette staples, 4 + 39 with rectangles; then U S^+."""
    return ((43.0 if c1 != 0.0 else 9.0) + 1.0) * MUL


def work(case):
    kind, v = case["kind"], float(_volume(case))
    links = 4.0 * v
    r = 4 if case.get("precision") in ("mixed", "fp32") else 8
    mat = 18.0 * r
    if kind in ("hmc", "batch"):
        c1 = case.get("c1", 0.0)
        fg = case.get("integrator", "leapfrog") == "force-gradient"
        forces = case["steps"] * (4 if fg else 1)
        # a shift reads U and writes U'; an update reads U' and reads and writes P and U
        per = 3.5 * mat if fg else 5.0 * mat
        ends = 2 * (2 * 144.0) + 144.0 + 2 * 144.0  # both Hamiltonians, the drawn momenta, the result
        return {"bytes": links * (forces * per + ends),
                "flops": links * forces * (_force_flops(c1) + 2.5 * MUL) + links * 2 * 3 * MUL}
    if kind == "force":
        return {"bytes": links * 2 * mat, "flops": links * _force_flops(case["c1"])}
    if kind == "flow":
        clover = 9.0 * MUL  # per link: six planes of a site, six products each
        per_step = links * (2 + 3 + 2 + 2 + 1) * mat
        return {"bytes": case["steps"] * per_step + links * mat + 8 * v,
                "flops": links * (case["steps"] * (3 * (_force_flops(case["c1"]) + 2.5 * MUL) + clover) + clover)}
    if kind == "measure":
        return {"bytes": links * mat + 2 * 8 * v, "flops": links * 9.0 * MUL}
    if kind == "topology":
        return {"bytes": links * mat + 40 * v, "flops": v * 7 * 36 * MUL}
    if kind == "adjoint":
        # forward stages, and per stage the pull-back: the force's derivative (36 products a link) and the local part
        n = 3.0 * case["steps"]
        return {"bytes": links * mat * n * (3.5 + 7.0),
                "flops": links * n * (_force_flops(0.0) + 2.5 * MUL + 46.0 * MUL)}
    # flowed: per step and flowed link the staple, its Jacobian and determinant, and the 18 pairs it enters
    n = len(_flow_steps(case))
    return {"bytes": links * mat * (3.0 * n + 2.0), "flops": v * n * 0.5 * (18 * 2000.0 + 20 * 1024.0)}


def tolerance(case):
    if case.get("precision") in ("mixed", "fp32"):
        # FP32 links: their rounding over a trajectory or a flow, in the sums taken of them (3e-7 seen), and in a
        # trajectory's difference of two energies (0.02 of some hundreds)
        return {"rel": 1e-4 if case["kind"] in ("hmc", "batch") else 4e-6}
    # FP64 throughout; energy differences of a trajectory lose the digits of the energies, and 40 flow steps leave
    # a small loss and gradient that carry the rounding of the way (2e-11 and 1.4e-12 seen)
    return {"rel": {"hmc": 1e-9, "batch": 1e-9, "adjoint": 1e-10}.get(case["kind"], 1e-12)}


# ---------------------------------------------------------------------------
# the same numbers in 64 bits from plain torch.  Fields have the shape
# (..., T, Z, Y, X, 4, 3, 3); a path is a list of directions, mu forward and
# -mu - 1 backward.

def _shape(u, case):
    return u.reshape(case["t"], case["z"], case["y"], case["x"], *u.shape[1:])


def _at(f, offsets, tail=2):
    """f(x + offsets) for a field with `tail` trailing dimensions."""
    dims = [mu for mu in range(4) if offsets[mu]]
    if not dims:
        return f
    return torch.roll(f, [-offsets[mu] for mu in dims], [f.dim() - tail - 1 - mu for mu in dims])


def _line(u, path, at=(0, 0, 0, 0)):
    at, out = list(at), None
    for d in path:
        mu = d if d >= 0 else -d - 1
        if d < 0:
            at[mu] -= 1
        m = _at(u[..., mu, :, :], at)
        m = m if d >= 0 else _dag(m)
        if d >= 0:
            at[mu] += 1
        out = m if out is None else _mm(out, m)
    return out


def _ta(m):
    a = (m - _dag(m)) / 2
    tr = a.diagonal(dim1=-1, dim2=-2).sum(-1) / 3
    return a - tr[..., None, None] * torch.eye(3, dtype=a.dtype, device=a.device)


def _tr(m):
    return m.diagonal(dim1=-1, dim2=-2).sum(-1).real


def _trp(a, b):
    """tr(a b), real part."""
    return (a * b.transpose(-1, -2)).sum((-1, -2)).real


def _staple(u, mu, c1):
    s = 0
    for nu in range(4):
        if nu == mu:
            continue
        for e in (nu, -nu - 1):
            b = -e - 1
            s = s + (1 - 8 * c1) * _line(u, [e, mu, b])
            if c1 != 0.0:
                s = s + c1 * (_line(u, [e, e, mu, b, b]) + _line(u, [e, mu, mu, b, -mu - 1])
                              + _line(u, [-mu - 1, e, mu, mu, b]))
    return s


def _force(u, beta, c1):
    """beta: a number, or a tensor that broadcasts over a field's matrices."""
    return torch.stack([-beta / 3 * _ta(_mm(u[..., mu, :, :], _dag(_staple(u, mu, c1)))) for mu in range(4)], -3)


def _action(u, beta, c1, dims):
    p = r = 0.0
    for mu in range(4):
        for nu in range(4):
            if mu < nu:
                p = p + (_tr(_line(u, [mu, nu, -mu - 1, -nu - 1])) - 3).sum(dims)
            if mu != nu and c1 != 0.0:
                r = r + (_tr(_line(u, [mu, mu, nu, -mu - 1, -mu - 1, -nu - 1])) - 3).sum(dims)
    return -beta / 3 * ((1 - 8 * c1) * p + c1 * r)


def _evolve(u, p, eps):
    return _mm(_exp(eps * p), u)


def _trajectory(u, p, beta, c1, steps, integrator, lattice=(-7, -6, -5, -4)):
    """(links, delta_h) after molecular dynamics of unit length; `beta` broadcasts over leading dimensions."""
    scalars = tuple(d + 3 for d in lattice)
    wide = beta[:, None, None, None, None, None, None] if torch.is_tensor(beta) else beta
    energy = lambda: -_trp(p, p).sum((-5, -4, -3, -2, -1)) / 2 + _action(u, beta, c1, scalars)  # noqa: E731
    h0, dt = energy(), 1.0 / steps
    if integrator == "leapfrog":
        for _ in range(steps):
            u = _evolve(u, p, dt / 2)
            p = p + dt * _force(u, wide, c1)
            u = _evolve(u, p, dt / 2)
    else:
        lam, ttheta = 0.5 * (1 - 1 / math.sqrt(3.0)), (2 - math.sqrt(3.0)) / 48 * dt ** 3
        u = _evolve(u, p, lam * dt)
        for i in range(steps):
            for half in range(2):
                p = p + 0.5 * dt * _force(_evolve(u, _force(u, wide, c1), 4 * ttheta / dt), wide, c1)
                eps = (1 - 2 * lam) * dt if half == 0 else (2 * lam if i + 1 < steps else lam) * dt
                u = _evolve(u, p, eps)
    return u, energy() - h0


def _flow_step(u, eps, c1):
    z = 0.25 * _force(u, 3.0, c1)
    u = _evolve(u, z, eps)
    z = 8.0 / 9.0 * _force(u, 3.0, c1) - 17.0 / 9.0 * z
    u = _evolve(u, z, eps)
    return _evolve(u, 0.75 * _force(u, 3.0, c1) - z, eps)


def _leaf(u, mu, m, nu, n):
    a, b, ma, mb = mu, nu, -mu - 1, -nu - 1
    return (_line(u, [a] * m + [b] * n + [ma] * m + [mb] * n) + _line(u, [ma] * m + [mb] * n + [a] * m + [b] * n)
            + _line(u, [b] * n + [ma] * m + [mb] * n + [a] * m) + _line(u, [mb] * n + [a] * m + [b] * n + [ma] * m)) / 4


def _planes(u, m=1, n=1):
    f = {}
    for mu in range(4):
        for nu in range(mu + 1, 4):
            c = _leaf(u, mu, m, nu, n)
            if m != n:
                c = (c + _leaf(u, mu, n, nu, m)) / 2
            f[mu, nu] = (c - _dag(c)) / 2
    return f


def _energy(f):
    return sum(-_trp(_ta(g), _ta(g)) for g in f.values())


def _charge(f):
    return -(-_trp(f[0, 2], f[1, 3]) + _trp(f[0, 3], f[1, 2]) + _trp(f[2, 3], f[0, 1])) / (4 * math.pi ** 2)


def _basis(m):
    return torch.stack([m[..., 0, 1].imag, m[..., 0, 1].real, (m[..., 0, 0].imag - m[..., 1, 1].imag) / 2,
                        m[..., 0, 2].imag, m[..., 0, 2].real, m[..., 1, 2].imag, m[..., 1, 2].real,
                        math.sqrt(3.0) / 2 * (m[..., 0, 0].imag + m[..., 1, 1].imag)], -1)


def _flowed_effective_action(u, case):
    """Action of the flowed field minus the log-determinants of the masked steps."""
    x = torch.meshgrid(*(torch.arange(n, device=u.device) for n in u.shape[:4]), indexing="ij")
    gens = _su3(torch.eye(8, dtype=torch.float64, device=u.device))
    ln_det = 0.0
    for mask, mu, eps, size in _flow_steps(case):
        c = 0
        for nu in range(4):
            if nu != mu:
                for e in (nu, -nu - 1):
                    c = c + _line(u, [e] * size + [mu] + [-e - 1] * size)
        on = (sum(k // size for k in x) % 2) == (mask % 2)
        link = u[..., mu, :, :]
        um, cd = link[on], _dag(c)[on]
        xm = -eps * _ta(_mm(um, cd))
        # su(3) matrices as 8 x 8: N_ab = (TA(T_b U C^+))_a, (ad X)_ab = ([X, T_b])_a
        n = _basis(_ta(_mm(_mm(gens, um[:, None]), cd[:, None]))).transpose(-1, -2)
        ad = _basis(_mm(xm[:, None], gens) - _mm(gens, xm[:, None])).transpose(-1, -2)
        one = torch.eye(8, dtype=torch.float64, device=u.device)
        j = one
        for k in range(20, 1, -1):
            j = one - ad @ j / k
        ln_det = ln_det + torch.linalg.slogdet(one - eps * (j @ n))[1].sum()
        new = link.clone()
        new[on] = _mm(_exp(xm), um)
        u = torch.stack([new if k == mu else u[..., k, :, :] for k in range(4)], -3)
    return _action(u, case["beta"], case["c1"], (0, 1, 2, 3)) - ln_det


def _gradient(u, fn):
    """sum_a (dfn/domega_a) T_a at U = exp(omega . T) u, omega = 0."""
    w = torch.zeros((*u.shape[:-2], 8), dtype=torch.float64, device=u.device, requires_grad=True)
    value = fn(u + _mm(_su3(w), u))
    value.backward()
    return value.item(), _su3(w.grad)


# The per-site random streams: SHA-256 of decimal counters appended to the parent's state (rng-state.cpp).

_PRIMES = [p for p in range(2, 312) if all(p % d for d in range(2, int(p ** 0.5) + 1))]


def _root_bits(p, k):
    lo = 0  # floor of the k-th root of p times 2^32
    for bit in range(36, -1, -1):
        if (lo + (1 << bit)) ** k <= p << (32 * k):
            lo += 1 << bit
    return lo & 0xFFFFFFFF


_K = [_root_bits(p, 3) for p in _PRIMES[:64]]
_H0 = [_root_bits(p, 2) for p in _PRIMES[:8]]


def _compress(state, words):
    """One SHA-256 block; eight state words and sixteen message words, each an int64 tensor or int below 2^32."""
    def rot(v, n):
        return ((v >> n) | (v << (32 - n))) & 0xFFFFFFFF
    w = list(words)
    a, b, c, d, e, f, g, h = state
    for i in range(64):
        if i >= 16:
            s0 = rot(w[i - 15], 7) ^ rot(w[i - 15], 18) ^ (w[i - 15] >> 3)
            s1 = rot(w[i - 2], 17) ^ rot(w[i - 2], 19) ^ (w[i - 2] >> 10)
            w.append((w[i - 16] + s0 + w[i - 7] + s1) & 0xFFFFFFFF)
        t = h + (rot(e, 6) ^ rot(e, 11) ^ rot(e, 25)) + ((e & f) ^ ((e ^ 0xFFFFFFFF) & g)) + _K[i] + w[i]
        t2 = (rot(a, 2) ^ rot(a, 13) ^ rot(a, 22)) + ((a & b) ^ (a & c) ^ (b & c))
        a, b, c, d, e, f, g, h = (t + t2) & 0xFFFFFFFF, a, b, c, (d + t) & 0xFFFFFFFF, e, f, g
    return [(x + y) & 0xFFFFFFFF for x, y in zip(state, (a, b, c, d, e, f, g, h))]


def _words(block):
    return [int.from_bytes(block[4 * i:4 * i + 4], "big") for i in range(16)]


def _split(state, name):
    """The stream (hash, bytes hashed) split from one at index 0."""
    text = b"[0] {" + name.encode() + b"}"
    text = text.ljust(-(-len(text) // 64) * 64)
    h, n = state
    for i in range(0, len(text), 64):
        h = _compress(h, _words(text[i:i + 64]))
    return h, n + len(text)


def _stream(*names):
    s = (_H0, 0)
    for name in names:
        s = _split(s, name)
    return s


def _counter_words(index, n_bytes):
    """The padded block of "[index]"; index an int64 tensor below 1000."""
    digits = 1 + (index >= 10).long() + (index >= 100).long()
    text = torch.zeros((index.numel(), 64), dtype=torch.int64, device=index.device)
    text[:, 0] = ord("[")
    rest, row = index.clone(), torch.arange(index.numel(), device=index.device)
    for k in range(3):
        on = digits > k
        text[row[on], (digits - k)[on]] = (rest % 10 + ord("0"))[on]
        rest = rest // 10
    text[row, digits + 1] = ord("]")
    text[row, digits + 2] = 0x80
    bits = 8 * (n_bytes + digits + 2)
    t = text.view(-1, 16, 4)
    w = list(((t[..., 0] << 24) | (t[..., 1] << 16) | (t[..., 2] << 8) | t[..., 3]).unbind(-1))
    w[15] = bits
    return w


def _site_gaussians(stream, sites, count, sigma):
    """`count` Gaussians of each site's stream split from `stream` (Marsaglia's polar method), (sites, count)."""
    text = b"".join(f"[0] {{{i}}}".encode().ljust(64) for i in range(sites))
    t = torch.from_numpy(np.frombuffer(text, dtype=np.uint8).reshape(sites, 16, 4).astype(np.int64)).cuda()
    words = ((t[..., 0] << 24) | (t[..., 1] << 16) | (t[..., 2] << 8) | t[..., 3]).unbind(-1)
    h = torch.stack([v.expand(sites) if torch.is_tensor(v) else torch.full((sites,), v, device="cuda")
                     for v in _compress(stream[0], words)], -1)
    n_bytes = stream[1] + 64
    out = torch.zeros((sites, count), dtype=torch.float64, device="cuda")
    index = torch.zeros(sites, dtype=torch.int64, device="cuda")
    cache, left = torch.zeros((sites, 3, 2), dtype=torch.int64, device="cuda"), torch.zeros_like(index)
    made, second = torch.zeros_like(index), torch.zeros(sites, dtype=torch.bool, device="cuda")
    fresh, v1 = torch.ones_like(second), torch.zeros(sites, dtype=torch.float64, device="cuda")
    while True:
        on = (made < count).nonzero()[:, 0]
        if not on.numel():
            return out * sigma
        index[on] += 1 + fresh[on].long()  # a pair's first draw counts itself and the pair
        fresh[on] = False
        need = on[left[on] == 0]
        have = on[left[on] > 0]
        word = torch.zeros((sites, 2), dtype=torch.int64, device="cuda")
        left[have] -= 1
        word[have] = cache[have, left[have]]
        if need.numel():
            new = torch.stack(_compress(list(h[need].unbind(-1)), _counter_words(index[need], n_bytes)), -1)
            cache[need], left[need] = new[:, :6].view(-1, 3, 2), 3
            word[need] = new[:, 6:]
        x = (word[:, 0].double() * 4294967296.0 + word[:, 1].double()) * 2.0 ** -64 * 2.0 - 1.0
        one, two = on[~second[on]], on[second[on]]
        v1[one] = x[one]
        second[one] = True
        second[two] = False
        r = v1[two] ** 2 + x[two] ** 2
        ok = (r < 1.0) & (r != 0)
        two, r = two[ok], r[ok]
        fac = torch.sqrt(-2.0 * torch.log(r) / r)
        out[two, made[two]], out[two, made[two] + 1] = x[two] * fac, v1[two] * fac
        made[two] += 2
        index[two] += 1  # the pair's second value is a call of its own
        fresh[two] = True


def _uniform(stream):
    """The first uniform of [0, 1) of a stream."""
    w = _compress(stream[0], _words(b"[1]\x80".ljust(56, b"\0") + (8 * (stream[1] + 3)).to_bytes(8, "big")))
    return (w[6] * 4294967296.0 + w[7]) * 2.0 ** -64


def _momenta(stream, sites):
    return _su3(_site_gaussians(stream, sites, 32, 1.0 / math.sqrt(2.0)).view(sites, 4, 8))


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        return _exact_batch(case, seed)
    v = _volume(case)
    u = _links(v, seed)
    if case.get("precision") == "fp32":
        u = torch.view_as_complex(torch.view_as_real(u).float().double())
    u = _shape(u, case)
    if kind == "hmc":
        products = v * case["steps"] * (4 if case["integrator"] == "force-gradient" else 1) * (8 if case["c1"] else 1)
        if products > 6e7:
            return None  # minutes
        rs = _stream(f"hmc-{seed}", "1")
        p = _shape(_momenta(_split(rs, "set_rand_gauge_momentum"), v), case)
        u, dh = _trajectory(u, p, case["beta"], case["c1"], case["steps"], case["integrator"])
        dh = dh.item()
        accepted = dh <= 0.0 or _uniform(_split(rs, "metropolis_accept")) <= math.exp(-dh)
        # delta_h of FP32 dynamics differs from this one by the rounding along the way, of no particular size
        return {"accepted": accepted, "delta_h": np.array([dh]) if case["precision"] == "fp64" else None,
                "links": u.reshape(v, 4, 3, 3)}
    if kind == "force":
        return _force(u, case["beta"], case["c1"]).reshape(v, 4, 3, 3)
    if kind == "flow":
        e = []
        for _ in range(case["steps"]):
            u = _flow_step(u, case["eps"], case["c1"])
            e.append(_energy(_planes(u)).mean().item())
        return {"energy": np.array(e), "charge": _charge(_planes(u)).reshape(v, 1), "links": u.reshape(v, 4, 3, 3)}
    if kind == "measure":
        plaq = sum(_tr(_line(u, [a, b, -a - 1, -b - 1])).sum() for a in range(4) for b in range(a + 1, 4))
        f = _planes(u)
        return {"plaq": np.array([(plaq / (18 * v)).item()]), "energy": _energy(f).reshape(v, 1), "charge": _charge(f).reshape(v, 1)}
    if kind == "topology":
        c5 = 1.0 / 20.0
        coef = [((19 - 55 * c5) / 9, 1, 1), ((1 - 64 * c5) / 9 / 16, 2, 2), ((-64 + 640 * c5) / 45 / 4, 1, 2),
                ((1 / 5 - 2 * c5) / 9, 1, 3), (c5 / 81, 3, 3)]
        return torch.stack([k * _charge(_planes(u, m, n)).reshape(v) for k, m, n in coef], -1)
    if kind == "adjoint":
        def loss(w):
            for _ in range(case["steps"]):
                w = checkpoint(_flow_step, w, case["eps"], 0.0, use_reentrant=False)
            return _action(w, case["beta"], 0.0, (0, 1, 2, 3))
        value, grad = _gradient(u, loss)
        return {"loss": np.array([value]), "grad": grad.reshape(v, 4, 3, 3)}
    _, grad = _gradient(u, lambda w: _flowed_effective_action(w, case))
    return -0.5 * grad.reshape(v, 4, 3, 3)


def _exact_batch(case, seed):
    sides, betas = _chain_sides(case), _chain_betas(case)
    u = _links(_volume(case), seed)
    dh, plaq, at = np.zeros(len(sides)), np.zeros(len(sides)), 0
    for n in sorted(set(sides)):
        chains = [c for c, s in enumerate(sides) if s == n]
        v = n ** 4
        w = u[at:at + v * len(chains)].view(len(chains), n, n, n, n, 4, 3, 3)
        at += v * len(chains)
        p = torch.stack([_momenta(_stream(f"batch-{seed}", f"chain-{c}"), v) for c in chains]).view(w.shape)
        beta = torch.tensor([betas[c] for c in chains], dtype=torch.float64, device="cuda")
        plaq[chains] = (1.0 - 3.0 / (18.0 * v) * _action(w, 1.0, 0.0, (1, 2, 3, 4))).cpu().numpy()
        dh[chains] = _trajectory(w, p, beta, 0.0, case["steps"], "leapfrog")[1].cpu().numpy()
    return {"delta_h": dh if case["precision"] == "fp64" else None, "plaq": plaq}
