"""Boundary transposes of the inviscid residual that need their own boundary states:
the moving isothermal wall, and the characteristic boundary with a supersonic
freestream over a subsonic and over a supersonic interior.

Central differences of calcResidual, as in test_gpu_adjoint_bc.py with its bounds:
1e-6 of the result plus 1e-9 of |adjoint| |direction| (kinks of the Rusanov flux,
rounding over the step).  The state's step is 1e-7, at the moving wall 1e-8: the 3D
case has a kink 1e-7 away (the CPU oracle's differences at steps 1e-6, 1e-7, 3e-8, 1e-8
are 10.756285, 10.756183, 10.7561564, 10.7561565, the adjoint 10.7561564).  The boundary
state's step is 1e-6."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

NAMES = ("rhoBound", "uBound", "vBound", "wBound", "pBound")
MOVING_WALL = 13  # isothermal no-slip wall that moves (BC_TYPE, include/global.hpp:63-78)


def _check(mesh, seed, base, u0, eps=1e-7, **kw):
    from fr_learn_b200 import Solver

    rng = np.random.default_rng(seed)
    make = lambda b: Solver(mesh, dtType=0, dt=1e-3, **b, **kw)  # noqa: E731
    s = make(base)
    x, d = s.get("pos_spts"), mesh.nDims
    w = [0.05 * np.prod(np.cos(2.1 * x + 0.9 * k), -1) for k in range(d + 2)]
    rho, v, p = 1 + w[0], [u0 + w[1], 0.1 + w[2], 0.02 + w[-2]][:d], 0.75 + w[-1]
    U = np.stack([rho, *(rho * q for q in v), p / 0.4 + 0.5 * rho * sum(q * q for q in v)], -1)
    gbar, delta, theta = rng.standard_normal(U.shape), rng.standard_normal(U.shape), rng.standard_normal(5)

    def res(sol, state):
        sol.set("U_spts", state)
        sol.calcResidual(0)
        return sol.get("divF_spts", 0)

    s.set("U_spts", U)
    ubar, tbar = s.residual_vjp(gbar, theta)
    fd = np.sum(gbar * (res(s, U + eps * delta) - res(s, U - eps * delta))) / (2 * eps)
    adj, scale = np.sum(ubar * delta), np.linalg.norm(ubar) * np.linalg.norm(delta)
    assert abs(fd - adj) <= 1e-6 * abs(adj) + 1e-9 * scale, (fd, adj, scale)
    eps = 1e-6
    R = [res(make({**base, **{n: base[n] + sg * eps * t for n, t in zip(NAMES, theta)}}), U) for sg in (1, -1)]
    dR = (R[0] - R[1]) / (2 * eps)
    fd, scale = np.sum(gbar * dR), np.linalg.norm(gbar) * max(np.linalg.norm(dR), 1.0)
    assert abs(fd - tbar) <= 1e-6 * abs(fd) + 1e-9 * scale, (fd, tbar)


def _mesh(d, bc):
    from fr_learn_b200 import box2d, box3d

    sides = ("xmin", "xmax", "ymin", "ymax") + (("zmin", "zmax") if d == 3 else ())
    name = "isothermal_noslip" if bc == MOVING_WALL else bc
    m = (box2d(5, 4, 0.0, 1.0, 0.0, 1.0, bcs=dict.fromkeys(sides, name), perturb=0.1, seed=1) if d == 2 else
         box3d(3, 2, 3, (0.0,) * 3, (1.0,) * 3, bcs=dict.fromkeys(sides, name), perturb=0.1, seed=2))
    if bc == MOVING_WALL:
        m.bc[m.bc == 9] = MOVING_WALL
    return m


@pytest.mark.parametrize("order, d", [(2, 2), (3, 2), (2, 3)])
def test_moving_isothermal_wall(order, d):
    base = dict(rhoBound=1.1, uBound=0.4, vBound=0.1, wBound=0.05, pBound=0.8)
    _check(_mesh(d, MOVING_WALL), 21, base, 0.35, eps=1e-8, order=order, TWall=1.0, RGas=0.75, uWall=0.3, vWall=-0.2,
           wWall=0.1)


@pytest.mark.parametrize("u0", [0.35, 2.1])
@pytest.mark.parametrize("order, d, riemann", [(2, 2, 1), (3, 2, 0), (2, 3, 0)])
def test_supersonic_characteristic_boundary(order, d, riemann, u0):
    base = dict(rhoBound=1.1, uBound=2.0, vBound=0.1, wBound=0.05, pBound=0.8)
    _check(_mesh(d, "char"), 22, base, u0, order=order, riemannType=riemann)
