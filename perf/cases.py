"""Performance cases of the library: the calls a simulation makes per time / Picard step.

Every case goes through the package's public calls with host arrays in and out, as the
reference's MGTimeStep does: old fields and sources in, assembly of every level, the
multigrid solve, the new fields back.  The meshes, boundary rules, physics and smoothing
counts are those of exfemus_b200/workloads.py and of the test and benchmark workloads;
draw() varies the element counts, the levels, the physics and the precision.

  heat       one equation: implicit or steady conduction with element sources (MGSolT),
             smoothed by Gauss-Seidel (FP64 or mixed) or by GMRES + ILU (the reference's
             default level solver)
  ns         one Picard step of a lid cavity (2D) or a channel (3D), Vanka smoothing
  bouss      one segregated step of the heated cavity: Navier-Stokes, then temperature
  adjoint    a gradient: forward solve, transposed solve, derivatives with respect to the
             element sources and the boundary data
  turb       one step of the channel with kappa and omega and their eddy viscosity
  fsi        time steps of the mesh displacement, one system per direction
  residual   a nonlinear residual: assembly at a given field, then b - A x on the host
"""
import ctypes as C

import numpy as np

import exfemus_b200 as ex
from exfemus_b200 import _lib, workloads


def listed():
    return [
        # the smallest workload: one conduction solve on 32 x 32 elements (latency and launches)
        dict(name="heat2d", kind="heat", dim=2, nx=4, ny=4, nz=1, nlev=4, solver="gs", prec="fp64", nu=2, dt=0.0),
        # the same system with the level solver that the reference's templates ship with
        dict(name="heat2d_gmres", kind="heat", dim=2, nx=4, ny=4, nz=1, nlev=4, solver="gmres", prec="fp64", nu=2,
             dt=0.0),
        # an implicit temperature step on the 3D channel's mesh, 64 x 16 x 16 hex27
        dict(name="heat3d_step", kind="heat", dim=3, nx=8, ny=2, nz=2, nlev=4, solver="gs", prec="fp64", nu=2,
             dt=0.1),
        # lid-driven cavity at Re 400, 128 x 128, one Picard step in plain FP64 ...
        dict(name="cavity2d_fp64", kind="ns", dim=2, nx=4, ny=4, nz=1, nlev=6, prec="fp64", nu=3, re=400.0),
        # ... and with the FP32 V-cycle inside the FP64 defect correction
        dict(name="cavity2d_mixed", kind="ns", dim=2, nx=4, ny=4, nz=1, nlev=6, prec="mixed", nu=3, re=400.0),
        # the 3D channel's third level on its own in FP64: an ordinary 3D step, 32 x 8 x 8
        dict(name="channel3d_fp64", kind="ns", dim=3, nx=8, ny=2, nz=2, nlev=3, prec="fp64", nu=3, re=50.0),
        # the benchmark's 3D channel, 64 x 16 x 16 hex27/hex8, mixed precision (the largest)
        dict(name="channel3d_mixed", kind="ns", dim=3, nx=8, ny=2, nz=2, nlev=4, prec="mixed", nu=3, re=100.0),
        # differentially heated cavity, 256 x 256, both equations, mixed precision
        dict(name="bouss2d_mixed", kind="bouss", dim=2, nx=4, ny=4, nz=1, nlev=7, prec="mixed", nu=3, ra=1e5),
        # gradient with 65,536 element sources and 64 modes of wall data, 256 x 256
        dict(name="adjoint2d", kind="adjoint", dim=2, nx=4, ny=4, nz=1, nlev=7, prec="fp64", nu=3, modes=64,
             ra=1e5),
        # turbulent channel step, 128 x 64: Navier-Stokes with eddy viscosity, kappa, omega
        dict(name="turb2d", kind="turb", dim=2, nx=4, ny=2, nz=1, nlev=6, prec="mixed", nu=2),
        # four steps of the moving mesh's dx and dy, 128 x 64
        dict(name="fsi2d_steps", kind="fsi", dim=2, nx=4, ny=2, nz=1, nlev=6, prec="fp64", nu=2, steps=4),
        # nonlinear residual of the 3D channel: assembly of every level and one product
        dict(name="residual3d", kind="residual", dim=3, nx=8, ny=2, nz=2, nlev=4, prec="fp64", nu=3, re=100.0),
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(lo * (hi / lo) ** rng.random()))

    def fine(c):  # elements of the finest level
        f = 1 << (c["nlev"] - 1)
        return c["nx"] * f * c["ny"] * f * (c["nz"] * f if c["dim"] == 3 else 1)

    while True:
        kind = rng.choice(["heat", "heat", "ns", "ns", "ns", "bouss", "adjoint", "turb", "fsi", "residual"])
        dim = rng.choice([2, 3]) if kind in ("heat", "ns", "residual") else 2
        c = dict(kind=kind, dim=dim, nz=1, prec=rng.choice(["fp64", "mixed"]))
        if dim == 3:
            c.update(nx=rng.randint(4, 8), ny=rng.randint(2, 3), nz=rng.randint(2, 3), nlev=rng.choice([2, 3, 3, 4]))
            most = 16384 if c["prec"] == "mixed" or kind != "ns" else 4096
        else:
            long = kind in ("turb", "fsi")  # on a 2 x 1 box
            c.update(nx=rng.randint(3, 6), ny=rng.randint(2, 3) if long else rng.randint(3, 6), nlev=rng.choice([3, 4, 5, 5, 6, 6, 7]))
            most = {"heat": 65536, "ns": 32768, "bouss": 65536, "adjoint": 65536, "turb": 16384, "fsi": 16384,
                    "residual": 65536}[kind]
        if kind == "heat":
            c.update(nu=rng.choice([1, 2, 3]), dt=rng.choice([0.0, 0.1, 0.01]), solver="gs")
            if rng.random() < 0.25:  # the ILU recurrences: up to 64 x 64 elements
                c.update(solver="gmres", prec="fp64", nu=2)
                most = 4096 if dim == 2 else 512
        elif kind in ("ns", "residual"):
            c.update(nu=3, re=float(log_int(10, 100 if dim == 2 else 50)))
            if kind == "residual":
                c.update(prec="fp64")
        elif kind == "bouss":
            c.update(nu=3, ra=float(log_int(1000, 100000)))
        elif kind == "adjoint":
            c.update(nu=3, prec="fp64", modes=log_int(4, 64), ra=float(log_int(10000, 100000)))
        elif kind == "turb":
            c.update(nu=2)
        else:
            c.update(nu=2, prec="fp64", steps=rng.randint(1, 4))
            c["nx"] += c["nx"] % 2  # the solid begins at an element boundary
        if most // 256 <= fine(c) <= most:
            return c


# ------------------------------------------------------------------- inputs
def _box(c):
    k = c["kind"]
    if c["dim"] == 3:
        return (0.0, 4.0, 0.0, 1.0, 0.0, 1.0)
    return (0.0, 2.0, 0.0, 1.0) if k in ("turb", "fsi") else (0.0, 1.0, 0.0, 1.0)


def _n0(c):
    return (c["nx"], c["ny"], c["nz"])[:c["dim"]]


def _cells(c):
    f = 1 << (c["nlev"] - 1)
    return tuple(n * f for n in _n0(c))


def _mg(c, smoother, **kw):
    prec = _lib.PREC_MIXED if c["prec"] == "mixed" else _lib.PREC_FP64
    return ex.mg_params(eps=1e-10, max_cycles=100, nu_pre=c["nu"], nu_post=c["nu"], smoother=smoother,
                        precision=prec, **kw)


def _waves(rng, n=4, top=3.0):
    """Amplitudes and wave numbers of a smooth random field."""
    return rng.uniform(-1.0, 1.0, n) / np.arange(1, n + 1), rng.uniform(0.5, top, (n, 3)), rng.uniform(0.0, 6.28, n)


def _field(waves, xyz):
    out = np.zeros(xyz[0].size)
    for a, k, f in zip(*waves):
        out += a * np.sin(sum(k[d] * xyz[d] for d in range(len(xyz))) * 2.0 + f)
    return out


def _sources(seed, nel):
    return workloads.lognormal_source(nel, seed=seed)


def _channel_flow(xyz, rng):
    """Parabolic inflow profile carried along the channel, with a smooth disturbance that
    vanishes on the walls and at the inlet."""
    x, y = xyz[0], xyz[1]
    prof = 4.0 * y * (1.0 - y)
    if len(xyz) == 3:
        prof = prof * 4.0 * xyz[2] * (1.0 - xyz[2])
    u = [prof * (1.0 + 0.02 * x * _field(_waves(rng), xyz))]
    for _ in range(len(xyz) - 1):
        u.append(0.02 * prof * x * _field(_waves(rng), xyz))
    return u


def _cavity_flow(xyz, rng, lid):
    """A recirculation that vanishes on the walls, and the lid's velocity on its interior."""
    x, y = xyz[0], xyz[1]
    bump = 16.0 * x * (1.0 - x) * y * (1.0 - y)
    a, b = rng.uniform(0.1, 0.3), rng.uniform(0.0, 0.1)
    u = a * bump * (2.0 * y - 1.0) * (1.0 + 0.2 * _field(_waves(rng), xyz)) + b * bump
    v = -a * bump * (2.0 * x - 1.0) * (1.0 + 0.2 * _field(_waves(rng), xyz))
    if lid:
        u[(y == 1.0) & (x > 0.0) & (x < 1.0)] = 1.0
    return [u, v]


def _ns_vector(vel, ndof):
    x = np.zeros(ndof)
    x[:sum(v.size for v in vel)] = np.concatenate(vel)
    return x


def _top_wall(xyz):
    """w_i = integral of the node's basis function over the side y = 1."""
    x, y = xyz[0], xyz[1]
    top = np.where(y == 1.0)[0]
    order = top[np.argsort(x[top])]
    xs = x[order]
    w = np.zeros(x.size)
    h = xs[2::2] - xs[:-2:2]
    np.add.at(w, order[:-2:2], h / 6.0)
    np.add.at(w, order[1::2], 4.0 * h / 6.0)
    np.add.at(w, order[2::2], h / 6.0)
    return w


def _heat_data(c, seed, xyz):
    """Sources, the old temperature (zero on the walls) of a heat case."""
    q = _sources(seed, int(np.prod(_cells(c))))
    told = np.ones(xyz[0].size)
    b = _box(c)
    for d in range(c["dim"]):
        told *= (xyz[d] - b[2 * d]) * (b[2 * d + 1] - xyz[d])
    return q, told * (1.0 + 0.3 * _field(_waves(np.random.default_rng(seed)), xyz))


def _adjoint_data(c, seed, xyz):
    q = _sources(seed, int(np.prod(_cells(c))))
    rng = np.random.default_rng(seed)
    g = 0.1 * rng.standard_normal(c["modes"]) / np.arange(1, c["modes"] + 1)
    g[0] = 1.0
    told = workloads.t_initial(dict(box=_box(c)), xyz, xyz[0].size, g_modes=g)
    w = _top_wall(xyz) * (1.0 + 0.2 * _field(_waves(rng), xyz))
    return q, told, w


def prepare(case, seed):
    c = dict(case)
    kind = c["kind"]
    rng = np.random.default_rng(seed)
    mesh = ex.Mesh(c["dim"], c["nlev"], _n0(c), _box(c))
    xyz = mesh.xyz()
    s = dict(case=c, mesh=mesh)
    if kind in ("heat", "adjoint"):
        t = ex.MGSolT(mesh)
        if kind == "heat":
            t.GenBc(_lib.BC_HEAT_DIRICHLET)
            t.phys = ex.phys(inv_re=1.0, inv_prdl=1.0, inv_dt=1.0 / c["dt"] if c["dt"] > 0.0 else 0.0)
            s["q"], s["told"] = _heat_data(c, seed, xyz)
            smoother = _lib.SMOOTH_GMRES_ILU if c["solver"] == "gmres" else _lib.SMOOTH_GS
            s["mg"] = _mg(c, smoother)
        else:
            t.GenBc(_lib.BC_BOUSS_T)
            t.phys = ex.phys(**workloads.bouss_phys(dict(ra=c["ra"], pr=0.71))[1])
            s["q"], s["told"], s["w"] = _adjoint_data(c, seed, xyz)
            s["mg"] = _mg(c, _lib.SMOOTH_GS)
        s["t"] = t
    elif kind in ("ns", "residual"):
        ns = ex.MGSolNS(mesh)
        if c["dim"] == 3:
            ns.GenBc(_lib.BC_CHANNEL)
            vel, omega = _channel_flow(xyz, rng), 0.5 if c["nlev"] == 4 else 0.4
        else:
            ns.GenBc(_lib.BC_CAVITY)
            vel, omega = _cavity_flow(xyz, rng, True), 0.4
        ns.phys = ex.phys(inv_re=1.0 / c["re"])
        s["ns"], s["mg"] = ns, _mg(c, _lib.SMOOTH_VANKA, omega=omega)
        s["old"] = _ns_vector(vel, ns.ntop_dof)
    elif kind == "bouss":
        ns, t = ex.MGSolNS(mesh), ex.MGSolT(mesh)
        ns.GenBc(_lib.BC_BOUSS_NS)
        t.GenBc(_lib.BC_BOUSS_T)
        p_ns, p_t = workloads.bouss_phys(dict(ra=c["ra"], pr=0.71, inv_dt=1.0))
        ns.phys, t.phys = ex.phys(**p_ns), ex.phys(**p_t)
        ns.couple(t)
        t.couple(ns)
        s["old"] = _ns_vector([0.3 * v for v in _cavity_flow(xyz, rng, False)], ns.ntop_dof)
        x, y = xyz
        s["told"] = (1.0 - x) * (1.0 + 0.2 * x * _field(_waves(rng), xyz))
        s["ns"], s["t"] = ns, t
        s["mg"] = _mg(c, _lib.SMOOTH_VANKA, omega=0.4)
        s["mg_t"] = _mg(c, _lib.SMOOTH_GS)
    elif kind == "turb":
        ph = ex.phys(inv_re=0.01, inv_dt=10.0)
        ns = ex.MGSolNS(mesh)
        ns.GenBc(_lib.BC_CHANNEL)
        ns.phys = ph
        x, y = xyz
        b0, b1 = np.ones(x.size, np.int32), np.zeros(x.size, np.int32)
        b1[np.abs(x - 2.0) < 1e-12] = 1
        inlet = np.abs(x) < 1e-12
        b0[inlet], b1[inlet] = 0, 1
        wall = (np.abs(y) < 1e-12) | (np.abs(y - 1.0) < 1e-12)
        b0[wall], b1[wall] = 0, 2
        dist = mesh.wall_dist(wall.astype(np.int32))
        kw = []
        for var in (0, 1):
            k = ex.MGSolTBK(mesh, var)
            k.set_bc(b0, b1)
            k.set_wall(dist, 0.01)
            k.phys = ph
            kw.append(k)
        for k, o in ((kw[0], kw[1]), (kw[1], kw[0])):
            k.couple(ns)
            k.couple(o)
            ns.couple(k)
        s["old"] = _ns_vector(_channel_flow(xyz, rng), ns.ntop_dof)
        s["kold"] = (0.01 + 0.02 * y * (1.0 - y)) * (1.0 + 0.2 * _field(_waves(rng), xyz))
        s["wold"] = (40.0 + 30.0 * (y - 0.5) ** 2) * (1.0 + 0.1 * _field(_waves(rng), xyz))
        s["kold"][wall] = 0.0
        s["ns"], s["kw"] = ns, kw
        s["mg"] = _mg(c, _lib.SMOOTH_VANKA, omega=0.4)
        s["mg_t"] = _mg(dict(c, prec="fp64"), _lib.SMOOTH_GS)
    elif kind == "fsi":
        ns = ex.MGSolNS(mesh)
        x, y = xyz
        amp = rng.uniform(0.2, 0.4)
        ns.set_xold(_ns_vector([amp * np.sin(1.5 * x) * (0.5 + y) + 0.02 * _field(_waves(rng), xyz),
                                amp * np.sin(1.5 * x + 1.0) * (0.5 + y) + 0.1], ns.ntop_dof))
        b0, b1 = np.ones(x.size, np.int32), np.zeros(x.size, np.int32)
        top = np.abs(y - 1.0) < 1e-12
        b0[top], b1[top] = 0, 1
        inlet = np.abs(x) < 1e-12
        b0[inlet], b1[inlet] = 0, 0
        b0[x > 1.0 + 1e-12] = 2
        b0[np.abs(x - 1.0) < 1e-12] = 4
        ds = []
        for a in range(2):
            d = ex.MGSolDS(mesh, a)
            d.set_bc(b0, b1)
            d.set_fields(0.005)
            d.couple(ns)
            ds.append(d)
        ds[1].couple(ds[0])
        s["ns"], s["ds"], s["mg"] = ns, ds, _mg(c, _lib.SMOOTH_GS)
        s["zero"] = np.zeros(x.size)
    return s


# --------------------------------------------------------------------- runs
def _ctx(fn, *a):
    rc = fn(*a)
    if rc != _lib.EXF_ERR_NOT_CONVERGED:
        _lib.check(rc)


def run(s):
    kind = s["case"]["kind"]
    if kind == "heat":
        t = s["t"]
        t.set_source(s["q"])
        t.set_xold(s["told"])
        t.set_x(s["told"])
        t.MGTimeStep(0.0, s["mg"])
        return t.x()
    if kind == "ns":
        ns = s["ns"]
        ns.set_xold(s["old"])
        ns.set_x(s["old"])
        ns.MGTimeStep(0.0, s["mg"])
        return ns.x()
    if kind == "residual":
        ns = s["ns"]
        ns.set_xold(s["old"])
        ns.assemble_all()
        return ns.resid(ns.nlev - 1, s["old"], ns.rhs())
    if kind == "bouss":
        ns, t = s["ns"], s["t"]
        ns.set_xold(s["old"])
        ns.set_x(s["old"])
        t.set_xold(s["told"])
        t.set_x(s["told"])
        ex.timestep_loop([ns, t], [s["mg"], s["mg_t"]], 1, strict=False)
        return dict(ns=ns.x(), t=t.x())
    if kind == "adjoint":
        t, L = s["t"], s["t"].L
        t.set_source(s["q"])
        t.set_xold(s["told"])
        t.set_x(np.zeros(t.ntop_dof))
        st = _lib.ExfSolveStats()
        djdq, djdg = np.zeros(s["q"].size), np.zeros(t.ntop_dof)
        _ctx(L.exf_adjoint_forward, t.h, C.byref(t.phys), C.byref(s["mg"]), C.byref(st))
        _ctx(L.exf_adjoint_backward, t.h, C.byref(t.phys), C.byref(s["mg"]), _lib.dptr(s["w"]), _lib.dptr(djdq),
             _lib.dptr(djdg), C.byref(st))
        return dict(t=t.x(), djdq=djdq, djdg=djdg)
    if kind == "turb":
        ns, (k, w) = s["ns"], s["kw"]
        for e, old in ((ns, s["old"]), (k, s["kold"]), (w, s["wold"])):
            e.set_xold(old)
            e.set_x(old)
        ex.timestep_loop([ns, k, w], [s["mg"], s["mg_t"], s["mg_t"]], 1, strict=False)
        return dict(ns=ns.x(), k=k.x(), w=w.x())
    for d in s["ds"]:
        d.set_xold(s["zero"])
        d.set_x(s["zero"])
    ex.timestep_loop(s["ds"], [s["mg"]] * 2, s["case"]["steps"], strict=False)
    return [d.x() for d in s["ds"]]


# --------------------------------------------------------------------- work
CYCLES = 10  # V-cycles to 1e-10 that work() counts: what these smoothers take at best


def work(case):
    """Bytes: the fields in and out, each level's matrix written by its assembly and read
    once per smoothing sweep and residual of CYCLES cycles (the direct coarse solve left
    out).  Flops: two per matrix entry read, and the element integrals."""
    c = dict(case)
    dim, kind = c["dim"], c["kind"]
    vb = 4 if c["prec"] == "mixed" else 8
    total = dict(bytes=0.0, flops=0.0)

    def system(flow, value_bytes, solves, assemblies):
        d = dim if flow else 1
        for lev in range(c["nlev"]):
            ne = [n << lev for n in _n0(c)]
            qq = float(np.prod([8.0 * n + 1 for n in ne]))
            nn = float(np.prod([2.0 * n + 1 for n in ne]))
            ql = float(np.prod([5.0 * n + 1 for n in ne])) if flow else 0.0
            entries = d * d * qq + 2 * d * ql
            index = 4 * (qq + ql)
            nq = 3 ** dim
            total["flops"] += assemblies * float(np.prod(ne)) * nq * nq * nq * 2 * (dim * dim + 4 * dim)
            total["bytes"] += assemblies * 8 * entries
            if lev == c["nlev"] - 1:
                total["bytes"] += 8 * 3 * d * nn * max(1, assemblies)
            if lev == 0:
                continue
            passes = solves * CYCLES * (2 * c["nu"] * (2 if lev < c["nlev"] - 1 else 1) + 1)
            total["bytes"] += passes * (value_bytes * entries + index + 3 * value_bytes * d * nn)
            total["flops"] += passes * 2 * entries

    if kind == "heat":
        system(False, vb, 1, 1)
    elif kind == "adjoint":
        system(False, 8, 2, 2)
    elif kind == "ns":
        system(True, vb, 1, 1)
    elif kind == "residual":
        system(True, 8, 0, 1)
    elif kind == "bouss":
        system(True, vb, 1, 1)
        system(False, vb, 1, 1)
    elif kind == "turb":
        system(True, vb, 1, 1)
        system(False, 8, 2, 2)
    else:
        system(False, 8, 2 * c["steps"], 2 * c["steps"])
    return total


# -------------------------------------------------------------------- exact
# Conduction on a box has a tensor-product operator: with the 1D quadratic mass and
# stiffness matrices of each axis (M_d, K_d) and their generalised eigenvectors the
# discrete system is solved directly in 64 bits.
def _lattice(c):
    """Node number of each lattice point [.., J, I]: the library numbers the level-0
    vertices first, then the points that appear on level 0, 1, ..., each in lattice order."""
    nlev, shape = c["nlev"], [2 * n + 1 for n in _cells(c)][::-1]
    idx = np.indices(shape)
    cls = np.full(shape, nlev)
    for lev in range(nlev - 1, -1, -1):
        cls[np.all(idx % (1 << (nlev - 1 - lev)) == 0, axis=0)] = lev + 1
    cls[np.all(idx % (1 << nlev) == 0, axis=0)] = 0
    number = np.empty(cls.size, np.int64)
    number[np.argsort(cls.ravel(), kind="stable")] = np.arange(cls.size)
    return number.reshape(shape)


def _axis(n, lo, hi):
    h = (hi - lo) / n
    M, K = np.zeros((2 * n + 1, 2 * n + 1)), np.zeros((2 * n + 1, 2 * n + 1))
    me = h / 30.0 * np.array([[4.0, 2.0, -1.0], [2.0, 16.0, 2.0], [-1.0, 2.0, 4.0]])
    ke = 1.0 / (3.0 * h) * np.array([[7.0, -8.0, 1.0], [-8.0, 16.0, -8.0], [1.0, -8.0, 7.0]])
    load = np.zeros((2 * n + 1, n))
    for e in range(n):
        at = slice(2 * e, 2 * e + 3)
        M[at, at] += me
        K[at, at] += ke
        load[at, e] = h / 6.0 * np.array([1.0, 4.0, 1.0])
    return M, K, load


def _along(mats, v):
    """mats[k] applied along axis k of v (None: the identity)."""
    for k, m in enumerate(mats):
        if m is not None:
            v = np.moveaxis(np.tensordot(m, v, axes=(1, k)), 0, k)
    return v


class _Conduction:
    """shift M T + k K T on the box, axes in lattice order (.., y, x)."""

    def __init__(self, c, shift, k, fixed):
        b = _box(c)
        self.ax = [_axis(n, b[2 * d], b[2 * d + 1]) for d, n in enumerate(_cells(c))][::-1]
        self.free = [slice(1, -1) if f else slice(None) for f in fixed[::-1]]
        self.shift, self.k = shift, k
        self.V, self.lam = [], []
        for (M, K, _), f in zip(self.ax, self.free):
            R = np.linalg.cholesky(M[f, f])
            W = np.linalg.solve(R, np.linalg.solve(R, K[f, f]).T)
            lam, Q = np.linalg.eigh((W + W.T) / 2.0)
            self.V.append(np.linalg.solve(R.T, Q))
            self.lam.append(lam)

    def mass(self, v):
        return _along([m for m, _, _ in self.ax], v)

    def apply(self, v):
        out = self.shift * self.mass(v)
        for k in range(len(self.ax)):
            out = out + self.k * _along([self.ax[j][1] if j == k else self.ax[j][0] for j in range(len(self.ax))], v)
        return out

    def sources(self, q):
        return _along([ld for _, _, ld in self.ax], q)

    def solve(self, rhs):
        """The free nodes' solution, zero elsewhere."""
        f = tuple(self.free)
        y = _along([v.T for v in self.V], rhs[f])
        s = self.shift + self.k * sum(lam.reshape([-1 if j == a else 1 for j in range(len(self.lam))])
                                      for a, lam in enumerate(self.lam))
        out = np.zeros(rhs.shape)
        out[f] = _along(self.V, y / s)
        return out


def exact(case, seed):
    c = dict(case)
    if c["kind"] not in ("heat", "adjoint"):
        return None
    number = _lattice(c)
    cells, b = _cells(c), _box(c)
    grids = np.meshgrid(*[b[2 * d] + (b[2 * d + 1] - b[2 * d]) * (np.arange(2 * n + 1) / (2.0 * n))
                          for d, n in enumerate(cells)][::-1], indexing="ij")[::-1]
    xyz = np.empty((c["dim"], number.size))
    for d in range(c["dim"]):
        xyz[d][number.ravel()] = grids[d].ravel()

    def nodes(v):
        out = np.empty(v.size)
        out[number.ravel()] = v.ravel()
        return out

    if c["kind"] == "heat":
        q, told = _heat_data(c, seed, xyz)
        shift = 1.0 / c["dt"] if c["dt"] > 0.0 else 0.0
        A = _Conduction(c, shift, 1.0, [True] * c["dim"])
        return nodes(A.solve(A.sources(q.reshape(cells[::-1])) + shift * A.mass(told[number])))
    q, told, w = _adjoint_data(c, seed, xyz)
    A = _Conduction(c, 0.0, 1.0 / (c["ra"] * 0.71) ** 0.5, [True, False])
    wall = told[number].copy()
    wall[:, 1:] = 0.0
    t = wall + A.solve(A.sources(q.reshape(cells[::-1])) - A.apply(wall))
    lam = A.solve(w[number])
    djdq = _along([ld.T for _, _, ld in A.ax], lam)
    djdg = np.zeros(wall.shape)
    djdg[:, 0] = (w[number] - A.apply(lam))[:, 0]
    return dict(t=nodes(t), djdq=djdq.ravel(), djdg=nodes(djdg))
