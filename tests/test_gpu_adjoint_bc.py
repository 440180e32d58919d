"""The inviscid residual's transpose with every boundary condition, each order's
tile and both Riemann solvers: gbar . d(divF) along a random direction of the state,
and of the boundary state (rho, u, v, w, p), by central differences of calcResidual.

The Rusanov flux has a kink where both sides' wave speeds are equal, and traces of
smooth data nearly are: a central difference is off by O(eps) there, per unit of
|adjoint| |direction| (measured 1.4e-2 eps on the CPU oracle, whose differences at
steps 1e-6, 1e-7, 1e-8 close in on the adjoint), and by 1e-16 / eps from rounding.
At the state's step 1e-7 both are near 1e-9; the bound is 1e-6 of the result plus
1e-9 of |adjoint| |direction|."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BCS = ["char", "sup_in", "sup_out", "sub_in", "sub_out", "slip_wall", "symmetry", "isothermal_noslip",
       "adiabatic_noslip"]
NAMES = ("rhoBound", "uBound", "vBound", "wBound", "pBound")


def _check(mesh, seed, **kw):
    from fr_learn_b200 import Solver

    rng = np.random.default_rng(seed)
    base = dict(rhoBound=1.1, uBound=0.4, vBound=0.1, wBound=0.05, pBound=0.8, TWall=1.0, RGas=0.75)
    make = lambda b: Solver(mesh, dtType=0, dt=1e-3, **{**b, **kw})  # noqa: E731
    s = make(base)
    x, d = s.get("pos_spts"), mesh.nDims
    w = [0.05 * np.prod(np.cos(2.1 * x + 0.9 * k), -1) for k in range(d + 2)]
    rho, v, p = 1 + w[0], [0.35 + w[1], 0.1 + w[2], 0.02 + w[-2]][:d], 0.75 + w[-1]
    U = np.stack([rho, *(rho * q for q in v), p / 0.4 + 0.5 * rho * sum(q * q for q in v)], -1)
    gbar, delta, theta = rng.standard_normal(U.shape), rng.standard_normal(U.shape), rng.standard_normal(5)

    def res(sol, state):
        sol.set("U_spts", state)
        sol.calcResidual(0)
        return sol.get("divF_spts", 0)

    s.set("U_spts", U)
    ubar, tbar = s.residual_vjp(gbar, theta)
    eps = 1e-7
    fd = np.sum(gbar * (res(s, U + eps * delta) - res(s, U - eps * delta))) / (2 * eps)
    adj, scale = np.sum(ubar * delta), np.linalg.norm(ubar) * np.linalg.norm(delta)
    assert abs(fd - adj) <= 1e-6 * abs(adj) + 1e-9 * scale, (fd, adj, scale)
    eps = 1e-6
    R = [res(make({**base, **{n: base[n] + sg * eps * t for n, t in zip(NAMES, theta)}}), U) for sg in (1, -1)]
    dR = (R[0] - R[1]) / (2 * eps)
    fd, scale = np.sum(gbar * dR), np.linalg.norm(gbar) * max(np.linalg.norm(dR), 1.0)
    assert abs(fd - tbar) <= 1e-6 * abs(fd) + 1e-9 * scale, (fd, tbar)


@pytest.mark.parametrize("riemann", [0, 1])
@pytest.mark.parametrize("bc", BCS)
def test_boundary_vjp_2d(bc, riemann):
    from fr_learn_b200 import box2d

    mesh = box2d(5, 4, 0.0, 1.0, 0.0, 1.0, bcs=dict.fromkeys(("xmin", "xmax", "ymin", "ymax"), bc), perturb=0.1, seed=1)
    _check(mesh, 11, order=2 + BCS.index(bc) % 4, riemannType=riemann)


@pytest.mark.parametrize("bc", BCS)
def test_boundary_vjp_3d(bc):
    from fr_learn_b200 import box3d

    sides = ("xmin", "xmax", "ymin", "ymax", "zmin", "zmax")
    mesh = box3d(3, 2, 3, (0.0,) * 3, (1.0,) * 3, bcs=dict.fromkeys(sides, bc), perturb=0.1, seed=2)
    _check(mesh, 12, order=1 + BCS.index(bc) % 4)
