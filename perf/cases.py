"""Performance cases of the level-set library: what a program has it do, through
its public entry points (felspa_b200.level_set, .batch and .learned).

A case is a dict of plain values.  Its "kind" says which calls one pass makes:

* "operators": the operator evaluations of a program that owns its time loop
  (explicit_time_derivative, local_left_right_gradients) and the scalars it
  prints (mass, deviation of |grad phi| from 1).
* "steps":     the host-driven loop of a reference driver, one
  LevelSetSurface.advance_time(dt, single step) call after another.
* "levelset":  LevelSetSurface.run_steps between two outputs: the field comes
  from the host, `steps` substeps with a fixed-count reinitialisation every
  `every` of them, the field goes back to the host.
* "coupled":   the level set inside a flow solver: every outer step hands over
  a new nodal velocity field (set_velocity_fe) and takes a few substeps.
* "reinit":    one reinitialisation to a band (ReinitSimulatorLDG defaults).
* "batch":     many independent uneven 2D problems advanced together.
* "network":   forward and parameter-gradient passes of the patch network of
  the learned reinitialisation over a batch of patches.

Fields live on the host in the library's interface (FP64 vectors); a program
that runs FP32 problems keeps them in 32 bits, so such fields are returned so.
`exact` restates each kind in 64-bit torch (dense per-cell operator matrices).
"""
import math

import numpy as np
import torch

from felspa_b200 import abi
from felspa_b200 import fields as F
from felspa_b200.batch import Batch
from felspa_b200.learned import MLP
from felspa_b200.level_set import LevelSetSurface, Mesh

PSEUDO = 5          # pseudo-steps of the fixed-count reinitialisation


# ----------------------------------------------------------------------
# the cases
# ----------------------------------------------------------------------
def listed():
    return [
        # the smallest call: one evaluation of every operator on a tiny mesh
        {"name": "operators_2d_32", "kind": "operators", "nx": 32, "ny": 32, "nz": 0, "p": 1, "basis": "Q",
         "prec": "fp64", "flow": "vortex"},
        # the reference's own slotted-disk test: FE_DGP(1), FP64, host-driven
        # steps, viscous reinitialisation with the 2D limiter every 10
        {"name": "zalesak_p1_fp64_128", "kind": "steps", "nx": 128, "ny": 128, "nz": 0, "p": 1, "basis": "P",
         "prec": "fp64", "flow": "rotation", "steps": 20, "every": 10, "visc": 6.28e-5},
        # production 2D run: degree 2, 256^2, viscous sweep, graph periods
        {"name": "disk_q2_fp32_256", "kind": "levelset", "nx": 256, "ny": 256, "nz": 0, "p": 2, "basis": "Q",
         "prec": "fp32", "flow": "rotation", "steps": 120, "every": 20, "visc": 1e-3, "band": 0},
        # highest degree, ragged 2D mesh, FP64, inviscid sweep with limiter
        {"name": "vortex_q3_fp64_233x190", "kind": "levelset", "nx": 233, "ny": 190, "nz": 0, "p": 3, "basis": "Q",
         "prec": "fp64", "flow": "vortex", "steps": 60, "every": 10, "visc": 0.0, "band": 0},
        # uneven batch: sizes 32..256, degrees 1..3, Fourier velocities
        {"name": "batch_48", "kind": "batch", "problems": 48, "nmin": 32, "nmax": 256, "prec": "fp32", "steps": 40,
         "every": 10},
        # the headline 3D run: degree-2 sphere in the deformation field, 64^3
        {"name": "sphere_q2_fp32_64", "kind": "levelset", "nx": 64, "ny": 64, "nz": 64, "p": 2, "basis": "Q",
         "prec": "fp32", "flow": "deformation", "steps": 120, "every": 10, "visc": 0.0, "band": 0},
        # the same physics in the FP64 mode on a ragged box
        {"name": "sphere_q2_fp64_45x37x50", "kind": "levelset", "nx": 45, "ny": 37, "nz": 50, "p": 2, "basis": "Q",
         "prec": "fp64", "flow": "deformation", "steps": 60, "every": 10, "visc": 0.0, "band": 0},
        # the largest: 128^3, developed plume rolls, reinitialised every 5
        {"name": "plume_q2_fp32_128", "kind": "levelset", "nx": 128, "ny": 128, "nz": 128, "p": 2, "basis": "Q",
         "prec": "fp32", "flow": "plume", "steps": 40, "every": 5, "visc": 0.0, "band": 0},
        # 3D in the reference's default basis (FE_DGP), the sweep restricted
        # to a narrow band around the interface
        {"name": "sphere_p2_fp32_60_band", "kind": "levelset", "nx": 60, "ny": 60, "nz": 60, "p": 2, "basis": "P",
         "prec": "fp32", "flow": "deformation", "steps": 60, "every": 10, "visc": 0.0, "band": 6},
        # coupled to a flow solver: new degree-2 nodal velocity every 20 steps
        {"name": "coupled_q2_fp32_48", "kind": "coupled", "nx": 48, "ny": 48, "nz": 48, "p": 2, "basis": "Q",
         "prec": "fp32", "fe_degree": 2, "outer": 3, "inner": 20},
        # redistancing of a distorted field with the reference's band loop
        {"name": "reinit_band_q2_fp32_56", "kind": "reinit", "nx": 56, "ny": 64, "nz": 48, "p": 2, "basis": "Q",
         "prec": "fp32", "coeff": 2.0},
        # one training-sized batch through the 2D patch network, both ways
        {"name": "network_2d_8192", "kind": "network", "dim": 2, "rows": 8192},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["operators", "steps", "levelset", "levelset", "levelset", "coupled", "reinit", "batch",
                       "network"])
    if kind == "network":
        dim = rng.choice([2, 2, 3])
        return {"kind": kind, "dim": dim, "rows": _log_int(rng, 130, 16384 if dim == 2 else 6000)}
    if kind == "batch":
        return {"kind": kind, "problems": rng.randint(6, 48), "nmin": rng.randint(24, 48),
                "nmax": rng.randint(128, 256), "prec": rng.choice(["fp32", "fp64"]), "steps": 10 * rng.randint(1, 4),
                "every": 10}
    three = rng.random() < (0.5 if kind in ("operators", "steps") else 0.65)
    c = {"kind": kind, "p": rng.randint(1, 2 if three else 3), "basis": rng.choice(["Q", "Q", "P"]),
         "prec": rng.choice(["fp32", "fp64"])}
    if three:
        top = {"operators": 24, "steps": 32, "levelset": 80, "coupled": 48, "reinit": 56}[kind]
        n = _log_int(rng, 10, top)
        c.update(nx=n, ny=max(8, n + rng.randint(-7, 7)), nz=max(8, n + rng.randint(-7, 7)))
    else:
        top = {"operators": 96, "steps": 128, "levelset": 400, "coupled": 256, "reinit": 256}[kind]
        n = _log_int(rng, 24, top)
        c.update(nx=n, ny=max(16, n + rng.randint(-20, 20)), nz=0)
    flow = "deformation" if three else rng.choice(["rotation", "vortex"])
    if kind == "operators":
        c.update(prec="fp64", flow=flow)
    elif kind == "steps":
        c.update(flow=flow, steps=10 * rng.randint(1, 2), every=10, visc=rng.choice([1e-3, 1e-4]))
    elif kind == "levelset":
        every = rng.choice([5, 10, 20])
        c.update(flow=rng.choice([flow, "plume"]) if three else flow, steps=every * rng.randint(2, 5), every=every,
                 visc=rng.choice([0.0, 1e-3]), band=rng.choice([0, 0, 6]))
    elif kind == "coupled":
        c.update(fe_degree=rng.randint(1, 2), outer=rng.randint(1, 3), inner=rng.randint(5, 20))
    elif kind == "reinit":
        c.update(coeff=round(rng.uniform(1.2, 2.0), 2))
    return c


# ----------------------------------------------------------------------
# inputs (made with torch / numpy alone; shared by prepare and exact)
# ----------------------------------------------------------------------
def _dim(case):
    return 3 if case["nz"] else 2


def _cells(case):
    return (case["nx"], case["ny"], case["nz"])[:_dim(case)]


def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _legendre(p, x):
    """orthonormal Legendre values and derivatives on [0, 1]: [mode][point]"""
    t = 2.0 * np.asarray(x, dtype=np.float64) - 1.0
    v, d = [], []
    for k in range(p + 1):
        c = np.polynomial.legendre.Legendre.basis(k)
        s = math.sqrt(2 * k + 1)
        v.append(s * c(t))
        d.append(2.0 * s * c.deriv()(t) if k else np.zeros_like(t))
    return np.array(v), np.array(d)


def _gauss(n):
    x, w = np.polynomial.legendre.leggauss(n)
    return 0.5 * (x + 1.0), 0.5 * w


def _distance(case, seed):
    """(function of the point coordinates, flow description): the interface
    and the flow of this seed"""
    rng = np.random.default_rng([seed, 77])
    dim = _dim(case)
    j = rng.uniform(-0.03, 0.03, 3)
    rad = float(rng.uniform(0.13, 0.17))
    flow = case.get("flow", "")
    if flow == "plume":
        amp = rng.uniform(-0.01, 0.01, 6)
        k = rng.integers(1, 5, (6, 2))

        def phi(x):
            h = 0.5 + j[0]
            for a, (u, v) in zip(amp, k):
                h = h + float(a) * torch.cos(2 * math.pi * (int(u) * x[0] + int(v) * x[1]))
            return x[2] - h
        return phi
    centre = [0.5 + j[0], 0.75 + j[1]] if dim == 2 else [0.35 + j[0], 0.36 + j[1], 0.34 + j[2]]
    if case["kind"] in ("coupled", "reinit"):
        centre, rad = [0.5 + v for v in j[:dim]], 0.3 + (rad - 0.15)

    def sphere(x):
        return torch.sqrt(sum((x[d] - centre[d]) ** 2 for d in range(dim))) - rad
    if dim == 2 and flow == "rotation":     # the slotted disk
        def phi(x):
            lo, hi = (centre[0] - 0.025, centre[1] + rad - 0.25), (centre[0] + 0.025, centre[1] + rad)
            q = [torch.maximum(lo[d] - x[d], x[d] - hi[d]) for d in range(2)]
            out = torch.sqrt(q[0].clamp(min=0) ** 2 + q[1].clamp(min=0) ** 2)
            box = torch.where(torch.maximum(q[0], q[1]) > 0, out, torch.maximum(q[0], q[1]))
            return torch.maximum(sphere(x), -box)
        return phi
    if case["kind"] == "reinit":            # same interface, not a distance function
        b = float(rng.uniform(0.2, 0.4))

        def phi(x):
            return sphere(x) * (1.0 + b * torch.sin(3.0 * x[0] + 2.0) * torch.cos(2.0 * x[1]))
        return phi
    return sphere


def _field(case, seed):
    """the velocity of this seed, as the library takes it"""
    s = 1.0 + 0.2 * float(np.random.default_rng([seed, 78]).uniform(-1, 1))
    flow = case["flow"]
    f = {"rotation": lambda: F.ccw_rotation(omega=2 * math.pi * s), "vortex": lambda: F.single_vortex(period=2.0),
         "deformation": lambda: F.deformation_3d(), "plume": lambda: F.plume_3d(0.5 * s)}[flow]()
    if flow in ("vortex", "deformation"):
        f.terms = [(c, s * a, fs) for c, a, fs in f.terms]
    return f


_T0 = {"plume": 40.0}   # 1 - exp(-t) is 1: the developed rolls


def _project(case, phi):
    """L2 projection of phi with QGauss(p+2): [z][y][x][mode], the modes of Q"""
    dim, p, n = _dim(case), case["p"], _cells(case)
    x, w = _gauss(p + 2)
    L, _ = _legendre(p, x)
    dev = _device()
    A = torch.tensor(L * w, device=dev)
    pts = [torch.tensor((np.arange(n[d])[:, None] + x[None, :]) / n[d], device=dev) for d in range(dim)]
    if dim == 2:
        X, Y = pts[0][None, :, None, :], pts[1][:, None, :, None]
        v = phi([X, Y]).expand(n[1], n[0], p + 2, p + 2)
        return torch.einsum("yxrq,br,aq->yxba", v, A, A).reshape(n[1], n[0], -1)[None].contiguous()
    out = torch.empty((n[2], n[1], n[0], (p + 1) ** 3), dtype=torch.float64, device=dev)
    X, Y = pts[0][None, None, :, None, None, :], pts[1][None, :, None, None, :, None]
    for z in range(0, n[2], 8):
        Z = pts[2][z:z + 8, None, None, :, None, None]
        v = phi([X, Y, Z]).expand(Z.shape[0], n[1], n[0], p + 2, p + 2, p + 2)
        out[z:z + 8] = torch.einsum("zyxsrq,cs,br,aq->zyxcba", v, A, A, A).reshape(Z.shape[0], n[1], n[0], -1)
    return out


def _modes(dim, p, basis):
    """Q-layout index of every mode of a cell, in the library's order"""
    r = range(p + 1)
    return [a + (p + 1) * (b + (p + 1) * c) for c in (r if dim == 3 else range(1)) for b in r for a in r
            if basis == "Q" or a + b + c <= p]


def _initial(case, seed):
    """the field of this seed as a host vector (FP64; 32-bit values for FP32 problems)"""
    q = _project(case, _distance(case, seed))
    v = q[..., _modes(_dim(case), case["p"], case["basis"])].reshape(-1)
    if case["prec"] == "fp32":
        v = v.float().double()
    return v.cpu()


def _host(v):
    """a host buffer the program keeps (page-locked where there is a GPU)"""
    return v.pin_memory() if torch.cuda.is_available() else v.clone()


def _lattices(case, seed):
    """the flow solver's nodal velocities of the outer steps"""
    n, dim, k = _cells(case), _dim(case), case["fe_degree"]
    rng = np.random.default_rng([seed, 79])
    base = F.deformation_3d() if dim == 3 else F.single_vortex()
    out = []
    for _ in range(case["outer"]):
        a, s = float(rng.uniform(0.8, 1.2)), rng.uniform(0.0, 0.3, dim)
        out.append(np.ascontiguousarray(F.fe_lattice(lambda x: a * base(x) + 0.1 * np.cos(x + s), n, k)))
    return out


def _patches(case, seed):
    """network input: patches of distorted distance functions over h, and output gradients"""
    rng = np.random.default_rng([seed, 80])
    dim, rows = case["dim"], case["rows"]
    h = 1.0 / rng.integers(64, 257, rows)
    slope = rng.uniform(0.7, 1.3, rows)
    n = rng.standard_normal((rows, dim))
    n *= (slope / np.linalg.norm(n, axis=1))[:, None]
    off = rng.uniform(-6.0, 6.0, rows)
    nb = 3 ** dim
    x = np.zeros((rows, nb, nb), dtype=np.float64)
    r = (-1, 0, 1)
    for cell, i in enumerate([(a, b, c) for c in (r if dim == 3 else (0,)) for b in r for a in r]):
        x[:, cell, 0] = off + sum(n[:, d] * (i[d] + 0.5) for d in range(dim))
        for d in range(dim):
            x[:, cell, 3 ** d] = n[:, d] / math.sqrt(12.0)
    x += 0.02 * rng.standard_normal(x.shape)
    x = np.concatenate([x.reshape(rows, -1), (64.0 * h)[:, None]], axis=1).astype(np.float32)
    return x, (rng.standard_normal((rows, nb)) / rows).astype(np.float32)


def _weights(dim, seed):
    rng = np.random.default_rng([seed, 81])
    w = [730 if dim == 3 else 82, 256, 256, 256, 256, 27 if dim == 3 else 9]
    out = []
    for a, b in zip(w[:-1], w[1:]):
        out += [rng.standard_normal((b, a)).ravel() * math.sqrt(1.5 / a), 0.05 * rng.standard_normal(b)]
    return np.concatenate(out).astype(np.float32)


def _batch_size(case, i):
    """cells per axis of problem i: log-uniform over the case's range"""
    return int(round(case["nmin"] * (case["nmax"] / case["nmin"]) ** ((i + 0.5) / case["problems"])))


def _batch_instances(case, seed):
    """uneven problems, degrees 1..3 in turn: unions of circles in Fourier velocities"""
    out = []
    for i in range(case["problems"]):
        rng = np.random.default_rng([seed, 82, i])
        n = _batch_size(case, i)
        s = int(rng.integers(1 << 30))
        c = {"kind": "batch", "nx": n, "ny": n, "nz": 0, "p": 1 + i % 3, "basis": "Q", "prec": case["prec"]}
        cs = [(rng.uniform(0.2, 0.8, 2), float(rng.uniform(0.05, 0.2))) for _ in range(int(rng.integers(1, 5)))]

        def phi(x, cs=cs):
            ds = [torch.sqrt((x[0] - float(p[0])) ** 2 + (x[1] - float(p[1])) ** 2) - r for p, r in cs]
            v = ds[0]
            for d in ds[1:]:
                v = torch.minimum(v, d)
            return v
        out.append((c, phi, F.fourier_stream_2d(seed=s, sample=64)))
    return out


# ----------------------------------------------------------------------
# what a program has in hand, and one pass
# ----------------------------------------------------------------------
def _surface(case, cfl=0.1):
    n = _cells(case)
    return LevelSetSurface(Mesh(len(n), n), case["p"], basis=abi.BASIS_Q if case["basis"] == "Q" else abi.BASIS_P,
                           precision=abi.FP32 if case["prec"] == "fp32" else abi.FP64, cfl_max=cfl)


def _reinit_opts(case):
    kw = {}
    if case.get("visc"):
        kw.update(viscosity=case["visc"], cfl_max=0.1)
    if case.get("band"):
        kw.update(narrow_band=1, band_cells=float(case["band"]))
    return abi.default_reinit_opts(mode=abi.REINIT_FIXED, n_pseudo_steps=PSEUDO, **kw)


def prepare(case, seed):
    s = {"case": case}
    if case["kind"] == "network":
        s["net"] = MLP(dim=case["dim"])
        s["net"].set_params(_weights(case["dim"], seed))
        s["x"], s["dy"] = _patches(case, seed)
        return s
    if case["kind"] == "batch":
        inst = _batch_instances(case, seed)
        b = Batch([Mesh(2, (c["nx"], c["ny"])) for c, _, _ in inst], [c["p"] for c, _, _ in inst],
                  precision=abi.FP32 if case["prec"] == "fp32" else abi.FP64, cfl_max=0.1)
        s["phi0"], s["out"] = [], []
        for pb, (c, phi, vel) in zip(b.problems, inst):
            pb.set_velocity(vel)
            v = _project(c, phi).reshape(-1)
            s["phi0"].append(_host((v.float().double() if case["prec"] == "fp32" else v).cpu()).numpy())
            s["out"].append(_host(torch.zeros(pb.n_dofs, dtype=torch.float64)))
        s["field"] = torch.zeros(b.n_dofs, dtype=torch.float32 if case["prec"] == "fp32" else torch.float64)
        s["batch"] = b
        s["control"] = abi.default_ls_opts(reinit_frequency=case["every"], reinit=_reinit_opts(case))
        return s
    ls = _surface(case)
    s["ls"] = ls
    s["phi0"] = _host(_initial(case, seed)).numpy()
    s["out"] = _host(torch.zeros(ls.n_dofs, dtype=torch.float64))
    s["field"] = torch.zeros(ls.n_dofs, dtype=torch.float32) if case["prec"] == "fp32" else s["out"]
    if case["kind"] == "coupled":
        s["velocity"] = [_host(torch.from_numpy(v)).numpy() for v in _lattices(case, seed)]
    elif case["kind"] == "reinit":
        ls.reinit_simulator.control = abi.default_reinit_opts(band_width_coeff=case["coeff"])
    else:
        ls.problem.set_velocity(_field(case, seed))
        if "every" in case:
            ls.control = abi.default_ls_opts(reinit_frequency=case["every"], reinit=_reinit_opts(case))
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "network":
        return {"y": s["net"].forward(s["x"]), "grad": s["net"].backward(s["x"], s["dy"])}
    if kind == "batch":
        b = s["batch"]
        for pb, v in zip(b.problems, s["phi0"]):
            pb.set_state(v)
        b.run_steps(case["steps"], s["control"])
        at = 0
        for pb, o in zip(b.problems, s["out"]):
            pb.get_state(o.numpy())
            s["field"][at:at + pb.n_dofs].copy_(o)
            at += pb.n_dofs
        return s["field"]
    ls, pb = s["ls"], s["ls"].problem
    pb.set_state(s["phi0"])
    if kind == "operators":
        left, right = ls.reinit_simulator.local_left_right_gradients()
        return {"rate": ls.explicit_time_derivative(0.25), "left": left, "right": right,
                "mass": ls.integrate_mass(), "deviation": ls.gradient_deviation()}
    pb.set_time(_T0.get(case.get("flow"), 0.0))
    if kind == "steps":
        for _ in range(case["steps"]):
            ls.advance_time(1.0, True)
    elif kind == "levelset":
        ls.run_steps(case["steps"])
    elif kind == "coupled":
        for v in s["velocity"]:
            pb.set_velocity_fe(case["fe_degree"], v)
            ls.advance_steps(case["inner"])
    elif kind == "reinit":
        ls.reinit_simulator.run_iteration()
    pb.get_state(s["out"].numpy())
    if s["field"] is not s["out"]:
        s["field"].copy_(s["out"])
    return {"phi": s["field"], "t": ls.get_time()}


# ----------------------------------------------------------------------
# work of one pass
# ----------------------------------------------------------------------
def _sizes(dim, n, p, basis, prec):
    ncell = int(np.prod(n))
    return ncell, len(_modes(dim, p, basis)), 4 if prec == "fp32" else 8


def _step_work(dim, n, p, basis, prec, steps, pseudo, visc, point_wise=False):
    """SSP-RK3 substeps (8 state passes each: a read and a write per stage, and
    phi^n again in two of them) and HJ pseudo-steps (the field and phi0 read,
    the result written; with viscosity its diffusion term, with the 2D limiter
    one more pass); point_wise: the velocity at the quadrature points read per stage"""
    ncell, nb, s = _sizes(dim, n, p, basis, prec)
    n1, nq = p + 1, p + 2
    nm, nf = n1 ** dim, n1 ** (dim - 1)
    stage = ncell * (dim * dim * 2 * nm * n1 + dim * (2 * 2 * nm + (dim - 1) * 2 * 2 * nf * n1))
    point = ncell * nq ** dim * (2 * dim * n1 * 2 + 20 * dim)
    b = steps * 8 * s * ncell * nb + pseudo * (5 if dim == 2 else 3) * s * ncell * nb
    b += pseudo * (2 + 2 * dim) * s * ncell * nb if visc else 0
    if point_wise:
        b += steps * 3 * s * ncell * (dim * nq ** dim + dim * nq ** (dim - 1))
    return b, steps * 3 * stage + pseudo * point


def work(case):
    kind = case["kind"]
    if kind == "network":
        w = [730 if case["dim"] == 3 else 82, 256, 256, 256, 256, 27 if case["dim"] == 3 else 9]
        mac = sum(a * b for a, b in zip(w[:-1], w[1:]))
        io = case["rows"] * (w[0] + w[-1]) * 4
        return {"bytes": 3 * io + 8 * mac, "flops": 2 * case["rows"] * mac * 4}
    if kind == "batch":
        b = f = 0
        for i in range(case["problems"]):
            n = _batch_size(case, i)
            x, y = _step_work(2, (n, n), 1 + i % 3, "Q", case["prec"], case["steps"],
                              case["steps"] // case["every"] * PSEUDO, 0.0, True)
            b, f = b + x, f + y
        return {"bytes": b, "flops": f}
    n, dim = _cells(case), _dim(case)
    ncell, nb, s = _sizes(dim, n, case["p"], case["basis"], case["prec"])
    a = (dim, n, case["p"], case["basis"], case["prec"])
    host = 16 * ncell * nb
    if kind == "operators":
        b, f = _step_work(*a, 1, 1, 0.0)
        return {"bytes": 8 * ncell * nb * (2 + 2 * dim), "flops": f}
    if kind == "coupled":
        nodes = dim * np.prod([case["fe_degree"] * v + 1 for v in n])
        b, f = _step_work(*a, case["outer"] * case["inner"], 0, 0.0, True)
        return {"bytes": b + host + 8 * int(nodes) * case["outer"], "flops": f}
    if kind == "reinit":
        scale = (4.0 / (2.0 + case["p"]) ** 2 + 1.0) * (2 * case["p"] + 1)
        b, f = _step_work(*a, 0, int(math.ceil(case["coeff"] * scale / 0.2)), 0.0)
        return {"bytes": b + host, "flops": f}
    b, f = _step_work(*a, case["steps"], case["steps"] // case["every"] * PSEUDO, case["visc"])
    return {"bytes": b + host, "flops": f}


# ----------------------------------------------------------------------
# the same passes in 64-bit torch
# ----------------------------------------------------------------------
class _Exact:
    """DG level-set operators on the box [0,1]^dim in FP64: fields are
    [z][y][x][mode] in the Q layout (modes outside P stay zero), operators are
    dense per-cell matrices."""

    def __init__(self, dim, n, p, basis):
        self.dim, self.n, self.p = dim, tuple(n), p
        self.dev = _device()
        self.h = [1.0 / v for v in n]
        self.diam = math.sqrt(sum(v * v for v in self.h))
        self.x, self.w = _gauss(p + 2)
        keep = np.zeros((p + 1) ** dim)
        keep[_modes(dim, p, basis)] = 1.0
        self.keep = self._t(keep)
        self.L, self.D = _legendre(p, self.x)
        e, de = _legendre(p, np.array([0.0, 1.0]))
        self.E, self.dE = e, de                       # [mode][end]
        eye = np.eye(p + 1)
        # value and derivative matrices at the Gauss points (point <- mode)
        self.B = self._t(self._kron([self.L.T] * dim))
        self.G = [self._t(self._kron([self.D.T if a == d else self.L.T for a in range(dim)])) / self.h[d]
                  for d in range(dim)]
        self.wq = self._t(self._kron([self.w[:, None]] * dim)[:, 0])
        # at the vertices
        self.Bv = self._t(self._kron([e.T] * dim))
        self.Gv = [self._t(self._kron([de.T if a == d else e.T for a in range(dim)])) / self.h[d]
                   for d in range(dim)]
        # traces (face modes <- cell modes) on the lower / upper face of each
        # axis, their values at the face's Gauss points
        self.tr = [[self._t(self._kron([e[:, s][None, :] if a == d else eye for a in range(dim)]))
                    for s in range(2)] for d in range(dim)]
        self.Bf = self._t(self._kron([self.L.T] * (dim - 1)))
        self.wf = self._t(self._kron([self.w[:, None]] * (dim - 1))[:, 0])
        # K_ij = int L_j L_i' per axis, over h
        K = (self.D * self.w) @ self.L.T
        self.K = [self._t(self._kron([K if a == d else eye for a in range(dim)])) / self.h[d] for d in range(dim)]

    def _t(self, a):
        return torch.tensor(np.ascontiguousarray(a), dtype=torch.float64, device=self.dev)

    @staticmethod
    def _kron(ms):
        """axes x, y, z -> one matrix with x fastest"""
        out = ms[0]
        for m in ms[1:]:
            out = np.kron(m, out)
        return out

    def load(self, v):
        q = torch.zeros(tuple(self.n[::-1]) + (self.keep.numel(),), dtype=torch.float64, device=self.dev)
        if self.dim == 2:
            q = q[None]
        q[..., self.keep.bool()] = v.to(self.dev).reshape(q.shape[:3] + (-1,))
        return q

    def store(self, q):
        return q[..., self.keep.bool()].reshape(-1)

    def axis(self, d):
        return 2 - d

    # velocity -----------------------------------------------------------
    def set_velocity(self, f):
        """f([x, y, z]) -> components, at the cells' and faces' points and vertices"""
        self.face = []
        pts = [self._t((np.arange(m)[:, None] + self.x[None, :]) / m) for m in self.n]

        def grid(ps):
            out = []
            for d, q in enumerate(ps):
                v = [1] * (2 * self.dim)
                v[self.dim - 1 - d], v[2 * self.dim - 1 - d] = q.shape
                out.append(q.reshape(v))
            return out

        def full(v, ps):
            v = torch.as_tensor(v, dtype=torch.float64, device=self.dev)
            sh = [q.shape[0] for q in ps][::-1] + [q.shape[1] for q in ps][::-1]
            v = v.expand(sh).reshape(sh[:self.dim] + [-1])
            return v[None] if self.dim == 2 else v
        self.vol = [full(u, pts) for u in f(grid(pts))]
        for d in range(self.dim):
            ps = list(pts)
            ps[d] = self._t(np.arange(self.n[d] + 1)[:, None] / self.n[d])
            self.face.append(full(f(grid(ps))[d], ps))
        ends = [self._t(np.arange(m + 1)[:, None] / m) for m in self.n]
        u = f(grid(ends))
        self.vmax = math.sqrt(float(sum((full(c, ends) ** 2) for c in u).max())) / self.diam

    def rhs(self, q, ct):
        v = (q @ self.B.T) * self.wq
        R = sum((v * self.vol[d]) @ self.G[d] for d in range(self.dim)) * ct
        for d in range(self.dim):
            ax = self.axis(d)
            lo = (q @ self.tr[d][1].T) @ self.Bf.T      # upper-face trace of the cell below the face
            hi = (q @ self.tr[d][0].T) @ self.Bf.T      # lower-face trace of the cell above it
            first, last = hi.narrow(ax, 0, 1), lo.narrow(ax, self.n[d] - 1, 1)
            below, above = torch.cat([first, lo], ax), torch.cat([hi, last], ax)
            u = ct * self.face[d]
            fl = ((u * torch.where(u > 0, below, above) * self.wf) @ self.Bf) / self.h[d]
            R = R + fl.narrow(ax, 0, self.n[d]) @ self.tr[d][0] - fl.narrow(ax, 1, self.n[d]) @ self.tr[d][1]
        return R * self.keep

    def step(self, q, t, dt, time):
        s = q + dt * self.rhs(q, time(t))
        s = (s + dt * self.rhs(s, time(t + dt)) + 3.0 * q) * 0.25
        return ((s + dt * self.rhs(s, time(t + 0.5 * dt))) * 2.0 + q) / 3.0

    def scaling(self):
        return (4.0 / (2.0 + self.p) ** 2 + 1.0) * (2 * self.p + 1)

    # reinitialisation -----------------------------------------------------
    def gradients(self, q):
        """left and right LDG gradients per axis"""
        left, right = [], []
        for d in range(self.dim):
            ax, n = self.axis(d), self.n[d]
            lo, hi = q @ self.tr[d][1].T, q @ self.tr[d][0].T
            below = torch.cat([hi.narrow(ax, 0, 1), lo], ax)           # trace from below each face
            above = torch.cat([hi, lo.narrow(ax, n - 1, 1)], ax)
            for out, tr in ((left, below), (right, above)):
                g = -(q @ self.K[d].T) + (tr.narrow(ax, 1, n) @ self.tr[d][1]
                                          - tr.narrow(ax, 0, n) @ self.tr[d][0]) / self.h[d]
                out.append(g * self.keep)
        return left, right

    def sign(self, q, B, G):
        v = q @ B.T
        g2 = sum((q @ g.T) ** 2 for g in G)
        return v / torch.sqrt(v * v + self.diam ** 2 * g2)

    def speed(self, S, left, right):
        """largest characteristic speed over the vertices, over the diameter"""
        g = []
        for a, b in zip(left, right):
            a, b = a @ self.Bv.T, b @ self.Bv.T
            ap, am, bp, bm = a.clamp(min=0), -a.clamp(max=0), b.clamp(min=0), -b.clamp(max=0)
            g.append(torch.where(S >= 0, torch.where(ap > bm, ap, bm), torch.where(am > bp, am, bp)))
        nrm = torch.sqrt(sum(v * v for v in g))
        small = nrm <= np.finfo(np.float64).eps
        return float(torch.where(small, nrm, S.abs()).max()) / self.diam

    def diffusion(self, q, nu):
        beta = 1.0 / math.sqrt(self.dim)
        R = torch.zeros_like(q)
        for d in range(self.dim):
            ax, n = self.axis(d), self.n[d]

            def traces(v):
                lo, hi = v @ self.tr[d][1].T, v @ self.tr[d][0].T
                return torch.cat([hi.narrow(ax, 0, 1), lo], ax), torch.cat([hi, lo.narrow(ax, n - 1, 1)], ax)

            def lift(f):
                return (f.narrow(ax, 1, n) @ self.tr[d][1] - f.narrow(ax, 0, n) @ self.tr[d][0]) / self.h[d]
            below, above = traces(q)
            g = (-(q @ self.K[d].T) + lift(0.5 * (below + above) + beta * (above - below))) * self.keep
            below, above = traces(g)
            f = 0.5 * (below + above) - beta * (above - below)
            f.narrow(ax, 0, 1).zero_()
            f.narrow(ax, n, 1).zero_()
            R = R + nu * (lift(f) - g @ self.K[d].T)
        return R * self.keep

    def limit(self, q):
        """2D minmod detector and WENO reconstruction"""
        n1, nx, ny = self.p + 1, self.n[0], self.n[1]
        q = q[0]
        avg = q[..., 0]

        def shift(v, d, s, fill=0.0):
            out = torch.full_like(v, fill)
            ax, m = (1, nx) if d == 0 else (0, ny)
            out.narrow(ax, 0 if s > 0 else 1, m - 1).copy_(v.narrow(ax, 1 if s > 0 else 0, m - 1))
            return out
        one = torch.ones_like(avg)
        sides = [(0, -1), (0, 1), (1, -1), (1, 1)]
        have = [shift(one, d, s) > 0 for d, s in sides]
        # the detector: per vertex its two faces' neighbours
        flag = torch.zeros_like(one, dtype=torch.bool)
        vv = q @ self.Bv.T
        for v, (fa, fb) in enumerate([(0, 2), (2, 1), (0, 3), (1, 3)]):
            interp = 0.0
            for f in (fa, fb):
                d, s = sides[f]
                interp = interp + (shift(avg, d, s) - avg) * (0.5 * s * (1 if (v >> d) & 1 else -1))
            a, b = vv[..., v] - avg, 3.0 * interp
            mm = torch.where(torch.sign(a) == torch.sign(b), torch.sign(a) * torch.minimum(a.abs(), b.abs()),
                             torch.zeros_like(a))
            flag |= have[fa] & have[fb] & (a != mm)
        vol = self.h[0] * self.h[1]

        def at(sh):
            """value, gradient and Hessian matrices at the home Gauss points shifted by sh"""
            ax = []
            for d in range(2):
                t = 2.0 * (self.x - sh[d]) - 1.0
                m = [[math.sqrt(2 * k + 1) * (2.0 ** j) * (np.polynomial.legendre.Legendre.basis(k).deriv(j)(t)
                                                           if j else np.polynomial.legendre.Legendre.basis(k)(t))
                      for k in range(n1)] for j in range(3)]
                ax.append([np.array(v).T for v in m])
            k = self._kron
            gr = [self._t(k([ax[0][1], ax[1][0]])) / self.h[0], self._t(k([ax[0][0], ax[1][1]])) / self.h[1]]
            he = [self._t(k([ax[0][2], ax[1][0]])) / self.h[0] ** 2,
                  self._t(k([ax[0][1], ax[1][1]])) / (self.h[0] * self.h[1]),
                  self._t(k([ax[0][0], ax[1][2]])) / self.h[1] ** 2]
            return self._t(k([ax[0][0], ax[1][0]])), gr, he

        def smooth(v, gr, he):
            b = sum((v @ g.T) ** 2 for g in gr) @ (self.wq * vol) * vol
            if self.p >= 2:
                hs = [v @ m.T for m in he]
                # rows 0 and 1 of the Hessians at points 0 and 1: (0,.) twice, (1,.) once
                ls = hs[0][..., 0] ** 2 + hs[1][..., 0] ** 2 + hs[1][..., 0] ** 2 + hs[2][..., 0] ** 2 \
                    + hs[1][..., 1] ** 2 + hs[2][..., 1] ** 2
                b = b + ls * (self.wq.sum() * vol) * vol ** 3
            return b
        B0, gr, he = at((0, 0))
        gam = sum(m.double() for m in have) * 0.001
        w = [(1.0 - gam) / (1e-6 + smooth(q, gr, he)) ** 2]
        pol = [q @ B0.T]
        for (d, s), m in zip(sides, have):
            qn = torch.stack([shift(q[..., k], d, s) for k in range(q.shape[-1])], -1)
            B, gr, he = at((s, 0) if d == 0 else (0, s))
            w.append(torch.where(m, 0.001 / (1e-6 + smooth(qn, gr, he)) ** 2, torch.zeros_like(avg)))
            v = qn @ B.T
            pol.append(v - (v @ self.wq)[..., None] + avg[..., None])
        tot = sum(w)
        new = sum(p * (a / tot)[..., None] for p, a in zip(pol, w))
        new = ((new * self.wq) @ B0) * self.keep
        return torch.where(flag[..., None], new, q)[None]

    def sweep(self, q, opts):
        """opts: pseudo-steps (or coeff: the band loop), viscosity, CFL"""
        S, Sv = self.sign(q, self.B, self.G), self.sign(q, self.Bv, self.Gv)
        left, right = self.gradients(q)
        run = cum = 0.0
        it = 0
        while it < opts["pseudo"] if opts.get("pseudo") is not None else cum < opts["coeff"] * self.diam:
            run = max(run, self.speed(Sv, left, right))
            left, right = self.gradients(q)
            nu = opts.get("visc", 0.0)
            scale = (self.p + 1) ** 2 * run + nu * (self.p + 1) ** 4 / self.diam ** 2 if nu else self.scaling() * run
            dt = opts["cfl"] / scale
            a2 = d1 = 0.0
            for a, b in zip(left, right):
                a, b = a @ self.B.T, b @ self.B.T
                a2, d1 = a2 + (0.5 * (a + b)) ** 2, d1 + (a - b)
            H = S * (torch.sqrt(a2) - 1.0) + 0.5 * S.abs() * d1
            R = -((H * self.wq) @ self.B) * self.keep
            if nu:
                R = R + self.diffusion(q, nu)
            q = q + dt * R
            if self.dim == 2:
                q = self.limit(q)
            cum += dt
            it += 1
        return q


def _time(field):
    """time factor of a field of this file's cases (they start where it is largest)"""
    if field.time_kind == abi.T_COS:
        return lambda t: math.cos(field.ta * t + field.tb)
    if field.time_kind == abi.T_COSPI:
        return lambda t: math.cos(math.pi * (field.ta * t + field.tb))
    if field.time_kind == abi.T_ONE_MINUS_EXP:
        return lambda t: 1.0 - math.exp(-field.ta * t)
    return lambda t: 1.0


def _separable(field):
    """the field's spatial part from its terms"""
    fn = {abi.F_ONE: lambda a, b, x: torch.ones_like(x), abi.F_LIN: lambda a, b, x: a * x + b,
          abi.F_SIN: lambda a, b, x: torch.sin(a * x + b), abi.F_COS: lambda a, b, x: torch.cos(a * x + b),
          abi.F_SINSQ: lambda a, b, x: torch.sin(a * x + b) ** 2,
          abi.F_SINPI: lambda a, b, x: torch.sin(math.pi * (a * x + b)),
          abi.F_COSPI: lambda a, b, x: torch.cos(math.pi * (a * x + b)),
          abi.F_SINPISQ: lambda a, b, x: torch.sin(math.pi * (a * x + b)) ** 2}

    def f(x):
        out = [torch.zeros((), dtype=torch.float64, device=x[0].device) for _ in x]
        for comp, coeff, fs in field.terms:
            v = coeff
            for d, (kind, a, b) in enumerate(fs[:len(x)]):
                v = v * fn[kind](a, b, x[d])
            out[comp] = out[comp] + v
        return out
    return f


def _nodal(case, lattice, x_dev):
    """the continuous nodal field of one lattice, as a function of the points"""
    n, k, dim = _cells(case), case["fe_degree"], _dim(case)
    nodes = [0.0, 1.0] if k == 1 else [0.0, 0.5, 1.0]
    lat = torch.tensor(lattice, device=x_dev)

    def f(x):
        # per axis: cell index and Lagrange basis at the points, from the 1D coordinates
        mats = []
        for d in range(dim):
            t = x[d].reshape(-1) * n[d]
            c = torch.floor(t + 1e-9).clamp(max=n[d] - 1)
            u = t - c
            m = torch.zeros((t.numel(), k * n[d] + 1), dtype=torch.float64, device=x_dev)
            for a in range(k + 1):
                v = torch.ones_like(u)
                for b in range(k + 1):
                    if b != a:
                        v = v * (u - nodes[b]) / (nodes[a] - nodes[b])
                m[torch.arange(t.numel()), c.long() * k + a] += v
            mats.append(m)
        out = []
        for comp in range(dim):
            v = lat[comp]
            v = torch.einsum("zyx,ax,by,cz->cba", v, *mats) if dim == 3 else torch.einsum("yx,ax,by->ba", v, *mats)
            # [z cell][z pt][y cell]... -> cells first, points last
            cells = [x[d].shape[dim - 1 - d] for d in reversed(range(dim))]
            pts = [x[d].shape[2 * dim - 1 - d] for d in reversed(range(dim))]
            v = v.reshape([s for pair in zip(cells, pts) for s in pair])
            out.append(v.permute(list(range(0, 2 * dim, 2)) + list(range(1, 2 * dim, 2))))
        return out
    return f


def _exact_network(case, seed):
    dim = case["dim"]
    x, dy = _patches(case, seed)
    dev = _device()
    w = [x.shape[1], 256, 256, 256, 256, dy.shape[1]]
    p = torch.tensor(_weights(dim, seed), dtype=torch.float64, device=dev)
    at, par = 0, []
    for a, b in zip(w[:-1], w[1:]):
        par.append((p[at:at + a * b].reshape(b, a).requires_grad_(), p[at + a * b:at + a * b + b].requires_grad_()))
        at += a * b + b
    v = torch.tensor(x, dtype=torch.float64, device=dev)
    for i, (W, c) in enumerate(par):
        v = v @ W.T + c
        if i < 4:
            v = torch.nn.functional.gelu(v)
    flat = [t for wc in par for t in wc]
    g = torch.autograd.grad((v * torch.tensor(dy, dtype=torch.float64, device=dev)).sum(), flat)
    return {"y": v.detach(), "grad": torch.cat([t.reshape(-1) for t in g])}


def exact(case, seed):
    kind = case["kind"]
    if kind == "network":
        return _exact_network(case, seed)
    if kind == "batch":
        out = []
        for c, phi, vel in _batch_instances(case, seed):
            ex = _Exact(2, (c["nx"], c["ny"]), c["p"], "Q")
            v = _project(c, phi).reshape(-1)
            q = ex.load(v.float().double() if case["prec"] == "fp32" else v)
            ex.set_velocity(_separable(vel))
            dt = 0.1 / (ex.vmax * ex.scaling())
            for k in range(case["steps"]):
                q = ex.step(q, 0.0, dt, lambda t: 1.0)
                if (k + 1) % case["every"] == 0:
                    q = ex.sweep(q, {"pseudo": PSEUDO, "cfl": 0.2})
            out.append(ex.store(q))
        return torch.cat(out)
    if case.get("band"):
        return None     # which tiles a narrow-band sweep covers is the library's choice
    ex = _Exact(_dim(case), _cells(case), case["p"], case["basis"])
    q = ex.load(_initial(case, seed))
    if kind == "reinit":
        q = ex.sweep(q, {"coeff": case["coeff"], "cfl": 0.2})
        return {"phi": ex.store(q), "t": 0.0}
    if kind == "coupled":
        t = run = 0.0
        for lattice in _lattices(case, seed):
            ex.set_velocity(_nodal(case, lattice, ex.dev))
            run = max(run, ex.vmax)
            dt = 0.1 / (run * ex.scaling())
            for _ in range(case["inner"]):
                q = ex.step(q, t, dt, lambda t: 1.0)
                t += dt
        return {"phi": ex.store(q), "t": t}
    field = _field(case, seed)
    time = _time(field)
    ex.set_velocity(_separable(field))
    if kind == "operators":
        left, right = ex.gradients(q)
        x, w = _gauss(case["p"] + 1)
        L, D = _legendre(case["p"], x)
        dim = ex.dim
        B = ex._t(ex._kron([L.T] * dim))
        wq = ex._t(ex._kron([w[:, None]] * dim)[:, 0])
        y, eps = -(q @ B.T), 1.5 * ex.diam
        H = 0.5 * (1.0 + y / eps + torch.sin(y * math.pi / eps) / math.pi)
        H = torch.where(y > eps, torch.ones_like(H), torch.where(y < -eps, torch.zeros_like(H), H))
        g2 = sum((q @ (ex._t(ex._kron([D.T if a == d else L.T for a in range(dim)])) / ex.h[d]).T) ** 2
                 for d in range(dim))
        vol = float(np.prod(ex.h))
        return {"rate": ex.store(ex.rhs(q, time(0.25))), "left": torch.stack([ex.store(v) for v in left]),
                "right": torch.stack([ex.store(v) for v in right]), "mass": float((H @ wq).sum()) * vol,
                "deviation": float(((torch.sqrt(g2) - 1.0).abs() @ wq).sum()) * vol}
    t, run = _T0.get(case["flow"], 0.0), 0.0
    opts = {"pseudo": PSEUDO, "cfl": 0.1 if case["visc"] else 0.2, "visc": case["visc"]}
    for k in range(case["steps"]):
        run = max(run, abs(time(t)) * ex.vmax)
        dt = 0.1 / (run * ex.scaling())
        q = ex.step(q, t, dt, time)
        t += dt
        if (k + 1) % case["every"] == 0:
            q = ex.sweep(q, opts)
    return {"phi": ex.store(q), "t": t}
