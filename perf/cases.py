"""The work a user has this framework do, as cases that can be timed.

Five kinds of call:

* ``march``     a solution in (pinned) host memory advanced by ``steps`` main-loop
                iterations with one ``update_host`` call, as a host program that keeps
                the reference's U_spts array does; ``monitor`` adds the residual norm
                that the reference's main loop prints;
* ``residual``  one ``calcResidual_noalloc`` of a state in the caller's device memory, in
                double precision, as an outer Newton or time integrator wants it;
* ``adjoint``   a gradient of the wall pressure over a bump with respect to the initial
                state and the Mach number: forward run, objective, reverse sweep;
* ``ensemble``  many independent vortices of several orders and sizes, one graph launch
                per step, each case with its own CFL dt;
* ``operator``  the operator products of one gradient evaluation as dense GEMMs on
                the caller's FP32 device arrays.

Mixed-precision results are handed on as single precision, the precision that mode's
operators and fluxes have.  ``exact`` restates the scheme (flux reconstruction on Gauss
points, DG correction, Rusanov / Roe / LDG fluxes, RK4) in 64-bit torch on the structured
grids the cases use.
"""
import math
import random

import numpy as np
import torch

from fr_learn_b200 import FRG_FP64, FRG_MIXED, Ensemble, Solver, box2d, box3d, bump2d, concat_meshes

GAMMA = 1.4


def listed():
    return [
        # 2D advection of a Gaussian, the smallest grid of the benchmark, called step by step: the cost of a call
        march("advection2d_step", "advection", (32, 32), 3, "fp64", steps=1),
        # the benchmark's isentropic vortex, mixed precision, tuned, between two outputs
        march("vortex2d_mixed", "euler", (128, 128), 4, "mixed", steps=50, riemann=1, cfl=0.5, tuned=True),
        # the same physics on a large odd-sized grid in double precision
        march("vortex2d_fp64_large", "euler", (256, 251), 3, "fp64", steps=20, riemann=1, cfl=0.5, tuned=True),
        # 3D Euler in double precision with farfield and slip walls and the residual norm, as the reference runs it
        march("euler3d_walls_fp64", "euler", (16, 16, 16), 3, "fp64", steps=5, bc="far", cfl=0.5, monitor=True),
        # 3D Euler, periodic, mixed precision, odd sizes
        march("euler3d_mixed", "euler", (31, 29, 27), 3, "mixed", steps=10),
        # the Taylor-Green vortex at the benchmark's size
        march("taylor_green_mixed", "ns", (32, 32, 32), 3, "mixed", steps=10),
        # a walled 3D Navier-Stokes channel, double precision, ragged sizes
        march("channel3d_fp64", "ns", (13, 11, 9), 2, "fp64", steps=10, bc="channel"),
        # a 2D Navier-Stokes channel between isothermal walls, double precision
        march("channel2d_fp64", "ns", (75, 48), 4, "fp64", steps=20, bc="channel"),
        # one residual for an outer solver that owns the memory
        {"name": "residual2d_fp64", "kind": "residual", "pde": "euler", "nx": 48, "ny": 40, "nz": 0, "order": 4,
         "prec": "fp64", "riemann": 1, "bc": "periodic"},
        # gradients of the bump channel, checkpointed
        {"name": "adjoint_bump", "kind": "adjoint", "nx": 96, "ny": 32, "order": 3, "steps": 100, "every": 25},
        # a batch of uneven vortices
        {"name": "ensemble_mixed", "kind": "ensemble", "count": 24, "lo": 2, "hi": 5, "steps": 200},
        # operator products of a 3D P = 3 gradient
        {"name": "operators3d", "kind": "operator", "dims": 3, "order": 3, "elements": 32768},
    ]


def march(name, pde, n, order, prec, steps, riemann=0, bc="periodic", cfl=0.0, tuned=False, monitor=False):
    c = {"kind": "march", "pde": pde, "nx": n[0], "ny": n[1], "nz": n[2] if len(n) == 3 else 0, "order": order,
         "prec": prec, "steps": steps, "riemann": riemann, "bc": bc, "cfl": cfl, "tuned": tuned, "monitor": monitor}
    return dict({"name": name}, **c) if name else c


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["march2d", "march2d", "march3d", "march3d", "residual", "adjoint", "ensemble", "operator"])
    prec = rng.choice(["fp64", "mixed"])
    if kind == "march2d":
        pde = rng.choice(["advection", "euler", "euler", "ns"])
        order = rng.randint(2, 5)
        most = int(math.sqrt((1.6e6 if pde == "ns" else 4.0e6) / (4 * (order + 1) ** 2)))
        nx = _log_int(rng, 16, most)
        ny = max(8, int(nx * rng.uniform(0.5, 1.0)))
        steps = rng.choice([1, 5, 20]) if nx * ny < 4000 else 20
        if pde == "euler":
            return march(None, pde, (nx, ny), order, prec, steps, riemann=rng.randint(0, 1), cfl=rng.choice([0.0, 0.5]),
                         tuned=rng.random() < 0.5)
        return march(None, pde, (nx, ny), order, prec, steps, bc="channel" if pde == "ns" else "periodic")
    if kind == "march3d":
        pde = rng.choice(["euler", "ns"])
        order = rng.randint(1, 4)
        n = _log_int(rng, 6, int((8.0e6 / (5 * (order + 1) ** 3)) ** (1 / 3)))
        n3 = tuple(max(4, n + rng.randint(-2, 2)) for _ in range(3))
        return march(None, pde, n3, order, prec, rng.choice([1, 5, 10]),
                     bc=rng.choice(["periodic", "far"] if pde == "euler" else ["periodic", "channel"]),
                     cfl=0.5 if pde == "euler" and rng.random() < 0.5 else 0.0, monitor=rng.random() < 0.25)
    if kind == "residual":
        pde = rng.choice(["euler", "ns"])
        if rng.random() < 0.6:
            return {"kind": "residual", "pde": pde, "nx": _log_int(rng, 10, 60), "ny": _log_int(rng, 10, 60), "nz": 0,
                    "order": rng.randint(2, 5), "prec": "fp64", "riemann": rng.randint(0, 1), "bc": "periodic"}
        return {"kind": "residual", "pde": pde, "nx": rng.randint(4, 12), "ny": rng.randint(4, 12),
                "nz": rng.randint(4, 12), "order": rng.randint(1, 3), "prec": "fp64", "riemann": 0, "bc": "periodic"}
    if kind == "adjoint":
        nx = _log_int(rng, 24, 128)
        return {"kind": "adjoint", "nx": nx, "ny": max(8, nx // rng.randint(2, 4)), "order": rng.randint(2, 4),
                "steps": rng.randint(10, 80), "every": rng.choice([0, 10, 25])}
    if kind == "ensemble":
        lo = rng.randint(2, 4)
        return {"kind": "ensemble", "count": rng.randint(6, 24), "lo": lo, "hi": rng.randint(lo, 5),
                "steps": rng.randint(20, 200)}
    dims = rng.randint(2, 3)
    return {"kind": "operator", "dims": dims, "order": rng.randint(1, 3 if dims == 3 else 5),
            "elements": _log_int(rng, 500, 32768)}


# --------------------------------------------------------------------- inputs
def _dims(case):
    return 3 if case.get("nz") else 2


def _grid(case):
    return (case["nx"], case["ny"], case["nz"])[:_dims(case)]


def _fields(case):
    return 1 if case["pde"] == "advection" else _dims(case) + 2


def _problem(case, seed):
    """Mesh, solver parameters and the initial state as a function of position."""
    rng = np.random.default_rng(seed)
    d, n, pde, order = _dims(case), _grid(case), case["pde"], case["order"]
    kw = {"order": order, "precision": FRG_MIXED if case["prec"] == "mixed" else FRG_FP64,
          "riemannType": case["riemann"], "timeType": 4}
    bc = case["bc"]
    lo, hi, speed, bcs = -10.0, 10.0, 3.0, {}
    if pde == "advection":
        lo, hi, speed = -5.0, 5.0, math.sqrt(2.0)
        kw.update(equation=0, advectVx=1.0, advectVy=1.0, advectVz=1.0)
        x0 = rng.uniform(-2, 2, d)

        def state(x):
            return np.exp(-((x - x0) ** 2).sum(-1))[..., None]
    elif pde == "euler" and d == 2:
        kw.update(rhoBound=1.0, uBound=1.0, vBound=1.0, pBound=1.0)
        x0, eps = rng.uniform(-4, 4, 2), rng.uniform(2, 5)

        def state(x):
            r = np.mod(x - x0 + 10.0, 20.0) - 10.0
            f = 1.0 - (r ** 2).sum(-1)
            rho = (1 - eps ** 2 * (GAMMA - 1) / (8 * GAMMA * np.pi ** 2) * np.exp(f)) ** (1 / (GAMMA - 1))
            g = eps / (2 * np.pi) * np.exp(f / 2)
            return _conservative(rho, [1 - g * r[..., 1], 1 + g * r[..., 0]], rho ** GAMMA)
    elif pde == "euler":
        lo, hi, speed = 0.0, 1.0, 1.8
        kw.update(rhoBound=1.0, uBound=0.5, vBound=0.1, wBound=0.0, pBound=1 / GAMMA)
        if bc == "far":
            bcs = {k: "char" for k in ("xmin", "xmax", "ymin", "ymax")}
            bcs.update(zmin="slip_wall", zmax="slip_wall")
        a, ph = rng.uniform(0.02, 0.06, 5), rng.uniform(0, 2 * np.pi, (5, 3))

        def state(x):
            w = [a[k] * np.prod(np.sin(2 * np.pi * x + ph[k]), -1) for k in range(5)]
            return _conservative(1 + w[0], [0.5 + w[1], 0.1 + w[2], w[3]], (1 + w[4]) / GAMMA)
    elif bc == "channel":  # Navier-Stokes between isothermal walls, at Mach 0.3
        lo, hi, speed = 0.0, 1.0, 1.4
        kw.update(viscous=1, rhoBound=1.0, pBound=1 / GAMMA, mu_inf=1e-3, prandtl=0.72, TWall=1.0, RGas=1 / GAMMA)
        bcs = {"ymin": "isothermal_noslip", "ymax": "isothermal_noslip"}
        a, ph = rng.uniform(0.01, 0.03, 3), rng.uniform(0, 2 * np.pi, 3)

        def state(x):
            y = 4 * x[..., 1] * (1 - x[..., 1])
            w = [a[k] * y * np.sin(2 * np.pi * x[..., 0] + ph[k]) for k in range(3)]
            vel = [0.3 * y + w[0], w[1]] + ([w[2]] if d == 3 else [])
            return _conservative(1 + 0.3 * w[2], vel, np.full(y.shape, 1 / GAMMA))
    else:  # Navier-Stokes, periodic: Taylor-Green vortex at Mach 0.1
        lo, hi, speed = 0.0, 2 * np.pi, 11.0
        kw.update(viscous=1, mu_inf=1 / 1600, prandtl=0.71)
        ph = rng.uniform(0, 2 * np.pi, 3)

        def state(x):
            X = [x[..., k] + ph[k] for k in range(d)]
            cz, c2z = (np.cos(X[2]), np.cos(2 * X[2])) if d == 3 else (1.0, 1.0)
            p = 100 / GAMMA + (np.cos(2 * X[0]) + np.cos(2 * X[1])) * (c2z + 2) / 16
            vel = [np.sin(X[0]) * np.cos(X[1]) * cz, -np.cos(X[0]) * np.sin(X[1]) * cz] + [np.zeros_like(p)] * (d - 2)
            return _conservative(np.ones_like(p), vel, p)
    if case.get("cfl"):
        kw.update(dtType=1, CFL=case["cfl"])
    else:
        kw.update(dtType=0, dt=0.5 * (hi - lo) / max(n) / (speed * d * (order + 1) ** 2))
    flat = pde == "ns" and bc == "periodic"
    make = dict(bcs=bcs, perturb=0.0 if flat else 0.1, seed=seed % (1 << 31))
    mesh = box2d(*n, lo, hi, lo, hi, **make) if d == 2 else box3d(*n, (lo,) * 3, (hi,) * 3, **make)
    return mesh, kw, state


def _conservative(rho, vel, p):
    return np.stack([rho] + [rho * v for v in vel] + [p / (GAMMA - 1) + 0.5 * rho * sum(v * v for v in vel)], -1)


def _bump(case, seed):
    rng = np.random.default_rng(seed)
    mach, c = rng.uniform(0.4, 0.6), math.sqrt(GAMMA)
    mesh = bump2d(case["nx"], case["ny"], bc_top="symmetry")
    h = min(3.0 / case["nx"], 0.45 * 0.8 / case["ny"])
    kw = dict(order=case["order"], riemannType=1, timeType=4, dtType=0, rhoBound=1.0, uBound=mach * c, pBound=1.0,
              dt=0.5 * h / ((mach + 1) * c * 2 * (case["order"] + 1) ** 2))
    a, ph = rng.uniform(0.005, 0.02, 4), rng.uniform(0, 2 * np.pi, 4)

    def state(x):
        w = [a[k] * np.sin(2 * np.pi * x[..., 0] + ph[k]) * np.cos(np.pi * x[..., 1] / 0.8) for k in range(4)]
        return _conservative(1 + w[0], [mach * c + w[1], 0.1 * w[2]], 1 + w[3])

    return mesh, kw, state, np.array([0.0, c, 0.0, 0.0, 0.0])


def _vortices(case, seed):
    """The batch: sides and orders belong to the case, strengths, Mach numbers and meshes to the seed."""
    mix, rng = random.Random(case["count"] * 64 + case["lo"] * 8 + case["hi"]), np.random.default_rng(seed)
    groups = {}
    for k in range(case["count"]):
        side = mix.choice(range(16, 97, 8))
        order = case["lo"] + k % (case["hi"] - case["lo"] + 1)
        eps, ui = rng.uniform(1, 5), rng.uniform(0.1, 0.6) * math.sqrt(GAMMA / 2)

        def state(x, eps=eps, ui=ui):
            f = 1.0 - (x ** 2).sum(-1)
            rho = (1 - eps ** 2 * (GAMMA - 1) / (8 * GAMMA * np.pi ** 2) * np.exp(f)) ** (1 / (GAMMA - 1))
            g = eps / (2 * np.pi) * np.exp(f / 2)
            return _conservative(rho, [ui - g * x[..., 1], ui + g * x[..., 0]], rho ** GAMMA)

        groups.setdefault(order, []).append((side, (seed + 7919 * k) % (1 << 31), state))
    return groups


def _vortex_mesh(side, seed):
    return box2d(side, side, -10.0, 10.0, -10.0, 10.0, perturb=0.1, seed=seed)


# -------------------------------------------------------------------- the call
def prepare(case, seed):
    kind = case["kind"]
    if kind == "march":
        mesh, kw, state = _problem(case, seed)
        s = Solver(mesh, **kw)
        U0 = state(s.get("pos_spts"))
        if case["monitor"]:
            s.setMonitor(True)
        s.set("U_spts", U0)
        if case["tuned"]:
            s.autotune(5)
        U = torch.empty(U0.shape, dtype=torch.float64, pin_memory=True)
        U.numpy()[...] = U0
        return {"case": case, "s": s, "U": U}
    if kind == "residual":
        mesh, kw, state = _problem(case, seed)
        s = Solver(mesh, **kw)
        U = np.ascontiguousarray(state(s.get("pos_spts")).transpose(2, 0, 1))
        stream = torch.cuda.Stream()
        s.set_stream(stream.cuda_stream)
        U = torch.from_numpy(U).cuda()
        return {"case": case, "s": s, "stream": stream, "U": U, "divF": torch.empty_like(U)}
    if kind == "adjoint":
        mesh, kw, state, theta = _bump(case, seed)
        s = Solver(mesh, **kw)
        return {"case": case, "s": s, "U0": state(s.get("pos_spts")), "theta": theta}
    if kind == "ensemble":
        solvers = []
        for order, members in sorted(_vortices(case, seed).items()):
            union, grp = concat_meshes([_vortex_mesh(side, sd) for side, sd, _ in members])
            s = Solver(union, order=order, dtType=1, CFL=0.5, riemannType=1, timeType=4, precision=FRG_MIXED)
            s.set_groups(grp, len(members))
            x = s.get("pos_spts")
            U = np.empty((s.nSpts, s.nEles, 4))
            for g, (_, _, state) in enumerate(members):
                U[:, grp == g] = state(x[:, grp == g])
            s.set("U_spts", U)
            s.autotune(5)
            solvers.append(s)
        return {"case": case, "solvers": solvers, "ens": Ensemble(solvers)}
    d, order, n = case["dims"], case["order"], case["elements"]
    mesh = box2d(16, 8) if d == 2 else box3d(8, 4, 4)
    # a handle whose element count the arrays have: the product acts on the caller's arrays only
    mesh = type(mesh)(d, np.resize(mesh.xv, (n,) + mesh.xv.shape[1:]), *_row_of_cells(d, n))
    s = Solver(mesh, order=order, precision=FRG_MIXED)
    stream = torch.cuda.Stream()
    s.set_stream(stream.cuda_stream)
    g = torch.Generator(device="cuda").manual_seed(seed)
    ld = (n + 31) // 32 * 32
    shape = {"U": s.nSpts, "Dc": s.nFpts}
    X = {k: 1 + 0.1 * torch.randn((s.nFields, m, ld), generator=g, device="cuda") for k, m in shape.items()}
    out = {k: torch.empty((s.nFields, m, ld), device="cuda")
           for k, m in [("tr", s.nFpts)] + [("g%d" % q, s.nSpts) for q in range(d)]}
    torch.cuda.synchronize()
    return {"case": case, "s": s, "stream": stream, "X": X, "out": out, "n": n, "ld": ld}


def _row_of_cells(d, n):
    """Corner ids and boundary conditions of n cells that touch nowhere."""
    nc, nf = (4, 4) if d == 2 else (8, 6)
    return np.arange(n * nc, dtype=np.int32).reshape(n, nc), np.full((n, nf), 1, np.int32)


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "march":
        s, U = state["s"], state["U"]
        s.update_host(U.numpy(), case["steps"])
        out = {"U": U.float() if case["prec"] == "mixed" else U}
        if case["monitor"]:
            norm = s.getNormResidual(2)
            out["norm"] = norm.astype(np.float32) if case["prec"] == "mixed" else norm
        return out
    if kind == "residual":
        s, stream = state["s"], state["stream"]
        s.calcResidual_noalloc(state["U"].data_ptr(), state["divF"].data_ptr(), stream.cuda_stream)
        return state["divF"]
    if kind == "adjoint":
        s = state["s"]
        s.set("U_spts", state["U0"])
        s.adjoint_forward(case["steps"], case["every"])
        J, dJ = s.objective("wall_pressure")
        lam0, theta_bar = s.adjoint_backward(None, state["theta"])
        return {"J": J, "dJ": dJ, "lam0": lam0, "theta_bar": theta_bar}
    if kind == "ensemble":
        state["ens"].update(case["steps"])
        return [torch.from_numpy(s.get("U_spts")).float() for s in state["solvers"]]
    s, X, out, ld = state["s"], state["X"], state["out"], state["ld"]
    s.apply_operator(0, 0, X["U"].data_ptr(), out["tr"].data_ptr(), ld)
    for q in range(case["dims"]):
        g = out["g%d" % q].data_ptr()
        s.apply_operator(1, q, X["U"].data_ptr(), g, ld)
        s.apply_operator(4, q, X["Dc"].data_ptr(), g, ld, 1.0)
    return {k: v[:, :, :state["n"]] for k, v in out.items()}


# ------------------------------------------------------------------------ work
def _stage_work(d, order, nv, s, viscous):
    """Bytes and flops of one RK stage per element: stage state in and out, step-start state and running
    combination in double precision, metrics and face data once; operators by sum factorisation."""
    n1 = order + 1
    ns, nf = n1 ** d, 2 * d * n1 ** (d - 1)
    by = ns * nv * (2 * s + 16) + ns * (d * d + 1) * s + nf * (d + 1) * s + 4 * nf
    fl = ns * nv * (2 * d * n1 + 4 * d + 2 * d * d + 6) + nf * nv * (4 * n1 + 4) + 40 * ns + 100 * nf
    if viscous:
        fl += ns * nv * (2 * d * n1 + 4 * d + 2 * d * d) + nf * nv * (2 * d * n1 + 4 * d) + 80 * ns + 80 * nf
    return by, fl


def work(case):
    kind = case["kind"]
    if kind in ("march", "residual"):
        d, nv, s = _dims(case), _fields(case), 8 if case["prec"] == "fp64" else 4
        n = math.prod(_grid(case))
        by, fl = _stage_work(d, case["order"], nv, s, case["pde"] == "ns")
        dof = n * (case["order"] + 1) ** d * nv
        if kind == "march":
            return {"bytes": 4 * case["steps"] * n * by + 16 * dof, "flops": 4 * case["steps"] * n * fl}
        return {"bytes": n * (by - (order_pts(case) * nv) * (2 * s + 16)) + 16 * dof, "flops": n * fl}
    if kind == "adjoint":
        by, fl = _stage_work(2, case["order"], 4, 8, False)
        n = case["nx"] * case["ny"]
        # forward stage, then a reverse stage of about three times its arithmetic over the same arrays
        return {"bytes": 8 * case["steps"] * n * by, "flops": 16 * case["steps"] * n * fl}
    if kind == "ensemble":
        b = f = 0
        for order, members in _vortices(case, 0).items():
            by, fl = _stage_work(2, order, 4, 4, False)
            n = sum(side * side for side, _, _ in members)
            b, f = b + 4 * case["steps"] * n * by, f + 4 * case["steps"] * n * fl
        return {"bytes": b, "flops": f}
    d, n1, n = case["dims"], case["order"] + 1, case["elements"]
    ns, nf, nv = n1 ** d, 2 * d * n1 ** (d - 1), d + 2
    return {"bytes": 4 * nv * n * (ns + nf + nf + d * ns), "flops": 2 * nv * n * (ns * nf + d * ns * (ns + nf))}


def order_pts(case):
    return (case["order"] + 1) ** _dims(case)


# ---------------------------------------------------------- the scheme in 64 bits
class _Scheme:
    """Flux reconstruction on a structured grid, fields [nv, (z,) y, x, (k,) j, i] (elements, then points)."""

    def __init__(self, xv, n, order, kw, ends):
        """xv [nE][nodes][d] (element index x fastest), n elements per direction, ends[d] = (lo, hi) boundary
        names or None where the direction is periodic."""
        self.d, self.n, self.kw, self.ends = len(n), n, kw, ends
        d = self.d
        dev = "cuda" if torch.cuda.is_available() else "cpu"
        t = lambda a: torch.tensor(np.asarray(a, np.float64), device=dev)  # noqa: E731
        x, w = np.polynomial.legendre.leggauss(order + 1)
        self.w = t(w)
        lag, dlag = _lagrange(x, x)
        self.D, self.lo, self.hi = t(dlag), t(_lagrange(x, [-1.0])[0][0]), t(_lagrange(x, [1.0])[0][0])
        leg = np.polynomial.legendre
        c = np.zeros(order + 2)
        c[order], c[order + 1] = 0.5, 0.5
        self.gR = t(leg.legval(x, leg.legder(c)))
        c[order + 1] = -0.5
        self.gL = t((-1) ** order * leg.legval(x, leg.legder(c)))
        # nodes as a tensor grid, then positions and Jacobians by 1D interpolation
        m = round(xv.shape[1] ** (1 / d))
        quad = [(0, 0), (1, 0), (1, 1), (0, 1)]
        if d == 2:
            at = quad if m == 2 else [(0, 0), (2, 0), (2, 2), (0, 2), (1, 0), (2, 1), (1, 2), (0, 1), (1, 1)]
        else:
            at = [a + (k,) for k in (0, 1) for a in quad]
        X = np.empty((d,) + tuple(reversed(n)) + (m,) * d)
        grid = xv.reshape(tuple(reversed(n)) + xv.shape[1:])
        for k, a in enumerate(at):
            X[(slice(None),) + (slice(None),) * d + tuple(reversed(a))] = np.moveaxis(grid[..., k, :], -1, 0)
        nodes, X = np.linspace(-1, 1, m), t(X)
        val, der = (t(v) for v in _lagrange(nodes, x))
        self.x = self._map(X, [val] * d)
        self.JG, self.det = self._metric(X, [val] * d, [der] * d)
        self.vol = self._weigh(self.det).sum(tuple(range(d, 2 * d)))
        self.face = []  # per direction: (lo, hi) of unit normal (outward) and area
        for q in range(d):
            sides = []
            for end, sign in ((-1.0, -1.0), (1.0, 1.0)):
                ev, ed = (t(v) for v in _lagrange(nodes, [end]))
                G, _ = self._metric(X, [ev if p == q else val for p in range(d)], [ed if p == q else der for p in range(d)])
                N = G[q].squeeze(2 * d - q)
                dA = N.square().sum(0).sqrt()
                sides.append((sign * N / dA, dA))
            self.face.append(sides)
        self.bound = [torch.tensor(v, dtype=torch.float64, device=dev) for v in (
            kw.get("rhoBound", 1.0), kw.get("uBound", 0.2), kw.get("vBound", 0.0), kw.get("wBound", 0.0),
            kw.get("pBound", 0.7142857143))]
        self.wave = None

    def _axis(self, q):
        return 2 * self.d - q

    def _along(self, M, U, q):
        a = self._axis(q)
        return torch.movedim(torch.tensordot(U, M, ([a], [1])), -1, a)

    def _map(self, X, ops):
        for q, M in enumerate(ops):
            X = self._along(M, X, q)
        return X

    def _metric(self, X, val, der):
        J = torch.stack([self._map(X, [der[p] if p == q else val[p] for p in range(self.d)]) for q in range(self.d)], -1)
        J = torch.movedim(J, 0, -2)  # [..., x_i, xi_j]
        det = torch.linalg.det(J)
        G = torch.linalg.inv(J) * det[..., None, None]  # [..., xi_j, x_i]
        return G.permute(-2, -1, *range(2 * self.d)), det

    def _weigh(self, A):
        """A (no field axis) times the quadrature weights of its trailing point axes."""
        for q in range(self.d):
            A = A * self.w.reshape((-1,) + (1,) * q)
        return A

    # -- layouts
    def from_ref(self, U):
        """[point][element][field] -> fields first, on the device."""
        n1 = len(self.w)
        U = torch.as_tensor(U, dtype=torch.float64, device=self.w.device)
        U = U.reshape((n1,) * self.d + tuple(reversed(self.n)) + (-1,))
        return U.permute((2 * self.d,) + tuple(range(self.d, 2 * self.d)) + tuple(range(self.d)))

    def to_ref(self, U):
        d = self.d
        U = U.permute(tuple(range(1 + d, 1 + 2 * d)) + tuple(range(1, 1 + d)) + (0,))
        return U.reshape(len(self.w) ** d, math.prod(self.n), -1)

    def points(self):
        return self.to_ref(self.x).cpu().numpy()

    # -- physics
    def prim(self, U):
        v = U[1:-1] / U[0]
        return U[0], v, (GAMMA - 1) * (U[-1] - 0.5 * U[0] * (v * v).sum(0))

    def flux(self, U):
        """[d][nv, ...]"""
        if U.shape[0] == 1:
            return [U * (1.0, 1.0, 1.0)[q] for q in range(self.d)]
        _, v, p = self.prim(U)
        out = []
        for q in range(self.d):
            F = U * v[q]
            add = torch.zeros_like(F)
            add[1 + q], add[-1] = p, p * v[q]
            out.append(F + add)
        return out

    def viscous(self, U, g):
        """Viscous flux of a state and its gradient g[d][nv, ...], with the index slips of the 3D stress terms
        that the reference has."""
        kw, d = self.kw, self.d
        rho, v = U[0], U[1:-1] / U[0]
        e = U[-1] / rho - 0.5 * (v * v).sum(0)
        mu, kap = kw["mu_inf"], kw["mu_inf"] / kw["prandtl"] * GAMMA
        dv = [(g[q][1:-1] - g[q][0] * v) / rho for q in range(d)]  # dv[q][k] = d v_k / d x_q
        de = [(g[q][-1] - 0.5 * (v * v).sum(0) * g[q][0] - rho * (v * dv[q]).sum(0) - g[q][0] * e) / rho for q in range(d)]
        diag = sum(dv[q][q] for q in range(d)) / 3.0
        t = {(q, q): 2 * mu * (dv[q][q] - diag) for q in range(d)}
        t[0, 1] = mu * (dv[1][0] + dv[0][1])
        if d == 3:
            t[0, 2], t[1, 2] = mu * (dv[2][0] + dv[0][1]), mu * (dv[2][0] + dv[1][1])
        tau = lambda a, b: t[min(a, b), max(a, b)]  # noqa: E731
        out = []
        for q in range(d):
            mom = [-tau(q, k) for k in range(d)]
            if d == 3 and q == 0:
                mom[2] = -t[2, 2]
            energy = -(sum(v[k] * tau(q, k) for k in range(d)) + kap * de[q])
            out.append(torch.stack([torch.zeros_like(rho)] + mom + [energy]))
        return out

    def rusanov(self, L, R, n):
        if L.shape[0] == 1:
            vn = n.sum(0)
            return vn * 0.5 * (L + R) + 0.5 * vn.abs() * (L - R), vn.abs()
        eig = None
        F = 0
        for U in (L, R):
            rho, v, p = self.prim(U)
            e = (v * n).sum(0).abs() + (GAMMA * p / rho).clamp_min(0).sqrt()
            eig = e if eig is None else torch.maximum(eig, e)
            F = F + sum(f * n[q] for q, f in enumerate(self.flux(U)))
        return 0.5 * (F - eig * (R - L)), eig

    def roe(self, L, R, n):
        (rL, vL, pL), (rR, vR, pR) = self.prim(L), self.prim(R)
        hL, hR = (L[-1] + pL) / rL, (R[-1] + pR) / rR
        k = (rR / rL).sqrt()
        um, hm = (vL + k * vR) / (k + 1), (hL + k * hR) / (k + 1)
        usq, un = 0.5 * (um * um).sum(0), (um * n).sum(0)
        a2 = (GAMMA - 1) * (hm - usq)
        a = a2.sqrt()
        nL, nR = (vL * n).sum(0), (vR * n).sum(0)
        eps = 0.5 * ((nL - nR).abs() + ((GAMMA * pL / rL).sqrt() - (GAMMA * pR / rR).sqrt()).abs())
        lam = [x.abs() for x in (un, un + a, un - a)]
        lam = [torch.where(x < 2 * eps, x * x / (4 * eps).clamp_min(1e-300) + eps, x) for x in lam]
        c2, c3 = 0.5 * (lam[1] + lam[2]) - lam[0], 0.5 * (lam[1] - lam[2]) / a
        dU = R - L
        a5 = (GAMMA - 1) * (usq * dU[0] - (um * dU[1:-1]).sum(0) + dU[-1])
        a6 = un * dU[0] - (n * dU[1:-1]).sum(0)
        p1, p2 = c2 * a5 / a2 - c3 * a6, c3 * a5 - c2 * a6
        one = torch.ones_like(un)
        diss = lam[0] * dU + torch.stack([p1 * one, *(p1 * um[q] + p2 * n[q] for q in range(self.d)), p1 * hm + p2 * un])
        F = sum((f + g) * n[q] for q, (f, g) in enumerate(zip(self.flux(L), self.flux(R))))
        return 0.5 * (F - diss), None

    def ghost(self, name, U, n):
        rho, v, p = self.prim(U)
        if name in ("slip_wall", "symmetry"):
            w = v - 2 * (v * n).sum(0) * n
            return torch.cat([U[:1], rho * w, U[-1:]])
        if name == "isothermal_noslip":
            r = p / (self.kw["RGas"] * self.kw["TWall"])
            return torch.cat([r[None], torch.zeros_like(v), (p / (GAMMA - 1))[None]])
        rB, pB = self.bound[0], self.bound[4]
        vB = torch.stack(self.bound[1:1 + self.d]).reshape((-1,) + (1,) * (n.dim() - 1))
        nL, nB, cL, cB = (v * n).sum(0), (vB * n).sum(0), (GAMMA * p / rho).sqrt(), (GAMMA * pB / rB).sqrt()
        k = 2 / (GAMMA - 1)  # subsonic farfield: outgoing invariant from inside, incoming from outside
        RL, RB = nL + k * cL, nB - k * cB
        c = 0.25 * (GAMMA - 1) * (RL - RB)
        s = torch.where(nL < 0, rB ** GAMMA / pB, rho ** GAMMA / p)
        r = (c * c / GAMMA * s) ** (1 / (GAMMA - 1))
        w = torch.where(nL < 0, vB + (0.5 * (RL + RB) - nB) * n, v + (0.5 * (RL + RB) - nL) * n)
        return torch.cat([r[None], r * w, (c * c * r / GAMMA / (GAMMA - 1) + 0.5 * r * (w * w).sum(0))[None]])

    # -- faces: for direction q, element axis E, "hi" of element i meets "lo" of element i + 1
    def _meet(self, q, lo, hi, both, at_end):
        """both(hi of i, lo of i+1, normal of hi) on every face of direction q, as (per lo side, per hi side);
        at_end(side, trace, normal) on the boundary planes."""
        E = self.d - q
        (nlo, _), (nhi, _) = self.face[q]
        f_hi, f_lo = both(hi, torch.roll(lo, -1, E), nhi)
        f_lo = torch.roll(f_lo, 1, E)
        if self.ends[q] is not None:
            m = self.n[q]
            cut = lambda A, i: A.narrow(E, i, 1)  # noqa: E731
            a = at_end(0, cut(lo, 0), cut(nlo, 0))
            b = at_end(1, cut(hi, m - 1), cut(nhi, m - 1))
            f_lo = torch.cat([a, f_lo.narrow(E, 1, m - 1)], E)
            f_hi = torch.cat([f_hi.narrow(E, 0, m - 1), b], E)
        return f_lo, f_hi

    def traces(self, U, q):
        a = self._axis(q)
        return torch.tensordot(U, self.lo, ([a], [0])), torch.tensordot(U, self.hi, ([a], [0]))

    def _lift(self, g, face, q):
        return face.unsqueeze(self._axis(q)) * g.reshape((-1,) + (1,) * q)

    def residual(self, U):
        d, kw = self.d, self.kw
        T = [self.traces(U, q) for q in range(d)]
        F = self.flux(U)
        waves = []
        visc = kw.get("viscous", 0)
        if visc:
            gr = []
            for q in range(d):
                lo, hi = T[q]
                mean = lambda a, b, n: (0.5 * (a + b),) * 2  # noqa: E731
                c_lo, c_hi = self._meet(q, lo, hi, mean, lambda s, a, n, q=q: 0.5 * (a + self.ghost(self.ends[q][s], a, n)))
                gr.append(self._along(self.D, U, q) + self._lift(self.gR, c_hi - hi, q) + self._lift(self.gL, c_lo - lo, q))
            g = [sum(gr[b] * self.JG[b, a] for b in range(d)) / self.det for a in range(d)]
            F = [f + v for f, v in zip(F, self.viscous(U, g))]
        div = 0
        for q in range(d):
            lo, hi = T[q]
            Ft = sum(self.JG[q, k] * F[k] for k in range(d))
            t_lo, t_hi = self.traces(Ft, q)
            if visc:
                gt = [self.traces(x, q) for x in g]
                vis = []
                for s in (0, 1):
                    n = self.face[q][s][0]
                    Fv = self.viscous(T[q][s], [x[s] for x in gt])
                    vis.append(sum(f * n[k] for k, f in enumerate(Fv)))

            def inner(a, b, n, q=q):
                f, eig = (self.roe if kw.get("riemannType") else self.rusanov)(a, b, n)
                waves.append((q, eig))
                if visc:
                    f = f + 0.5 * (vis[1] - torch.roll(vis[0], -1, d - q)) + kw.get("tau", 1.0) * (a - b)
                return f, -f

            def outer(s, a, n, q=q):
                G = self.ghost(self.ends[q][s], a, n)
                f, eig = self.rusanov(a, G, n)
                waves.append((q, s, eig))
                if visc:
                    f = f + vis[s].narrow(d - q, 0 if s == 0 else self.n[q] - 1, 1) + kw.get("tau", 1.0) * (a - G)
                return f

            f_lo, f_hi = self._meet(q, lo, hi, inner, outer)
            j_lo, j_hi = f_lo * self.face[q][0][1] + t_lo, f_hi * self.face[q][1][1] - t_hi
            div = div + self._along(self.D, Ft, q) + self._lift(self.gR, j_hi, q) - self._lift(self.gL, j_lo, q)
        return div, waves

    # -- time steps
    def dt(self, U):
        if not self.kw["dtType"]:
            return self.kw["dt"]
        d = self.d
        if self.wave is None:  # every element's own traces, once
            self.wave = []
            for q in range(d):
                w = []
                for s, tr in enumerate(self.traces(U, q)):
                    rho, v, p = self.prim(tr)
                    w.append((v * self.face[q][s][0]).sum(0).abs() + (GAMMA * p / rho).sqrt())
                self.wave.append(w)
        limit = [1.393, 0.464, 0.235, 0.1453, 0.100, 0.0736][len(self.w) - 1]
        total = 0
        for q in range(d):
            for s in (0, 1):
                A = self.wave[q][s] * self.face[q][s][1]
                for k in range(d - 1):
                    A = A * self.w.reshape((-1,) + (1,) * k)
                total = total + A.sum(tuple(range(d, 2 * d - 1)))
        return float((self.kw["CFL"] * limit * 2 * self.vol / total).min())

    def keep_waves(self, waves):
        """A face keeps its Rusanov wave speed in the element it was made from (the lower index)."""
        for q, *s, eig in waves:
            if eig is None:
                continue
            E, m = self.d - 1 - q, self.n[q]
            if s:
                self.wave[q][s[0]] = self.wave[q][s[0]].clone()
                self.wave[q][s[0]].narrow(E, 0 if s[0] == 0 else m - 1, 1).copy_(eig)
                continue
            self.wave[q] = [w.clone() for w in self.wave[q]]
            self.wave[q][1].narrow(E, 0, m - 1).copy_(eig.narrow(E, 0, m - 1))
            if self.ends[q] is None:
                self.wave[q][0].narrow(E, 0, 1).copy_(eig.narrow(E, m - 1, 1))

    def step(self, U, dt):
        first, out, Y = None, U, U
        for a, b in ((0.5, 1 / 6), (0.5, 1 / 3), (1.0, 1 / 3), (0.0, 1 / 6)):
            R, waves = self.residual(Y)
            first = R if first is None else first
            out = out - b * dt * R / self.det
            Y = U - a * dt * R / self.det
        if self.wave is not None:
            self.keep_waves(waves)
        return out, first


def _lagrange(nodes, at):
    """Values and derivatives [at][node] of the Lagrange basis."""
    nodes, at = np.asarray(nodes, np.float64), np.asarray(at, np.float64)
    val, der = np.ones((len(at), len(nodes))), np.zeros((len(at), len(nodes)))
    for j in range(len(nodes)):
        for m in range(len(nodes)):
            if m == j:
                continue
            term = np.full(len(at), 1.0 / (nodes[j] - nodes[m]))
            for k in range(len(nodes)):
                if k not in (j, m):
                    term *= (at - nodes[k]) / (nodes[j] - nodes[k])
            der[:, j] += term
            val[:, j] *= (at - nodes[m]) / (nodes[j] - nodes[m])
    return val, der


def _ends(case):
    d = _dims(case)
    if case["bc"] == "far":
        return [("char", "char"), ("char", "char"), ("slip_wall", "slip_wall")]
    wall = ("isothermal_noslip",) * 2
    return [wall if case["bc"] == "channel" and q == 1 else None for q in range(d)]


def exact(case, seed):
    kind = case["kind"]
    if kind in ("march", "residual"):
        mesh, kw, state = _problem(case, seed)
        S = _Scheme(mesh.xv, _grid(case), case["order"], kw, _ends(case))
        U = S.from_ref(state(S.points()))
        if kind == "residual":
            return S.to_ref(S.residual(U)[0]).permute(2, 0, 1).contiguous()
        for _ in range(case["steps"]):
            U, first = S.step(U, S.dt(U))
        out = {"U": S.to_ref(U).contiguous()}
        if case["monitor"]:
            out["norm"] = S._weigh(first.square() / S.det).sum(tuple(range(1, 2 * S.d + 1)))
        return out
    if kind == "adjoint":
        mesh, kw, state, theta = _bump(case, seed)
        S = _Scheme(mesh.xv, (case["nx"], case["ny"]), case["order"], kw, [("char", "char"), ("slip_wall", "symmetry")])
        dt, keep = kw["dt"], []
        U = S.from_ref(state(S.points()))
        for _ in range(case["steps"]):
            keep.append(U)
            U = S.step(U, dt)[0]
        U = U.detach().requires_grad_()
        wall = S.traces(U, 1)[0][:, 0]
        J = (S.prim(wall)[2] * S.face[1][0][1][0] * S.w).sum()
        dJ = lam = torch.autograd.grad(J, U)[0]
        bar, free = 0.0, S.bound[1].clone().requires_grad_()
        S.bound[1] = free
        for Y in reversed(keep):
            Y = Y.detach().requires_grad_()
            lam, b = torch.autograd.grad(S.step(Y, dt)[0], (Y, free), lam)
            bar += float(b) * theta[1]
        return {"J": float(J.detach()), "dJ": S.to_ref(dJ).contiguous(), "lam0": S.to_ref(lam).contiguous(), "theta_bar": bar}
    if kind == "ensemble":
        out = []
        for order, members in sorted(_vortices(case, seed).items()):
            part = []
            for side, sd, state in members:
                kw = dict(riemannType=1, dtType=1, CFL=0.5)
                S = _Scheme(_vortex_mesh(side, sd).xv, (side, side), order, kw, [None, None])
                U = S.from_ref(state(S.points()))
                for _ in range(case["steps"]):
                    U = S.step(U, S.dt(U))[0]
                part.append(S.to_ref(U))
            out.append(torch.cat(part, 1))
        return out
    return _exact_operators(case, seed)


def _exact_operators(case, seed):
    """Dense operators from the 1D tables; flux points in the reference's order around an element."""
    state = prepare(case, seed)
    d, order, n = case["dims"], case["order"], state["n"]
    p, n1 = order, order + 1
    x = np.polynomial.legendre.leggauss(n1)[0]
    unit = box2d(3, 3) if d == 2 else box3d(3, 3, 3)
    S = _Scheme(unit.xv, (3,) * d, order, {}, [None] * d)
    lo, hi, D, gL, gR = (v.cpu().numpy() for v in (S.lo, S.hi, S.D, S.gL, S.gR))
    lines = []  # (direction, side, the line's point for parameter i)
    if d == 2:
        for k in range(n1):
            lines.append((1, 0, lambda i, k=k: k + n1 * i))
        for k in range(n1):
            lines.append((0, 1, lambda i, k=k: i + n1 * k))
        for k in range(n1):
            lines.append((1, 1, lambda i, k=k: p - k + n1 * i))
        for k in range(n1):
            lines.append((0, 0, lambda i, k=k: i + n1 * (p - k)))
    else:
        spec = [(2, 0, lambda a, b, i: a + n1 * b + n1 * n1 * i), (2, 1, lambda a, b, i: p - a + n1 * b + n1 * n1 * i),
                (0, 0, lambda a, b, i: i + n1 * a + n1 * n1 * b), (0, 1, lambda a, b, i: i + n1 * (p - a) + n1 * n1 * b),
                (1, 0, lambda a, b, i: p - a + n1 * i + n1 * n1 * b), (1, 1, lambda a, b, i: a + n1 * i + n1 * n1 * b)]
        for q, s, f in spec:
            for b in range(n1):
                for a in range(n1):
                    lines.append((q, s, lambda i, f=f, a=a, b=b: f(a, b, i)))
    ns = n1 ** d
    E, C = np.zeros((len(lines), ns)), np.zeros((d, ns, len(lines)))
    for f, (q, s, at) in enumerate(lines):
        for i in range(n1):
            E[f, at(i)] = (lo, hi)[s][i]
            C[q, at(i), f] = (gL, gR)[s][i]
    G = np.zeros((d, ns, ns))
    for s in range(ns):
        for q in range(d):
            i = s // n1 ** q % n1
            for k in range(n1):
                G[q, s, s + (k - i) * n1 ** q] = D[i, k]
    U, Dc = (state["X"][k][:, :, :n].double() for k in ("U", "Dc"))
    mul = lambda M, X: torch.matmul(torch.tensor(M, device=X.device), X)  # noqa: E731
    out = {"g%d" % q: mul(G[q], U) + mul(C[q], Dc) for q in range(d)}
    out["tr"] = mul(E, U)
    return out
