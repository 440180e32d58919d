"""The line kernels (one thread per coordinate line) against the oracle where
their block shape changes and at the edges of their tiles: meshes that pick the
widest, the middle and the narrowest shape of each order, with a last tile of a
few elements, walls and farfield boundaries, CFL and fixed dt.

Tolerances: FP64 agrees with the reference's algorithm to rounding (1e-12, the
bound of every FP64 parity test); the mixed mode's state to 1e-6 in the 2-norm."""
import numpy as np
import pytest

from conftest import relerr

pytestmark = pytest.mark.gpu

FAR = dict(xmin="char", xmax="char", ymin="char", ymax="char", zmin="slip_wall", zmax="slip_wall")
WALL3 = dict(ymin="isothermal_noslip", ymax="adiabatic_noslip")
NS = dict(viscous=1, mu_inf=0.01, prandtl=0.72, pBound=1 / 1.4, uBound=0.3, TWall=1.0, RGas=1 / 1.4)
# block shapes change at 74 tiles: 2431 = 76 x 32 - 1, 1331 = 83 x 16 + 3, 605 = 75 x 8 + 5
SIZES3 = {"wide": (17, 13, 11), "middle": (11, 11, 11), "narrow": (5, 11, 11), "tiny": (3, 4, 3)}
CASES = {}
for P in (1, 2, 3, 4):
    for size, n in SIZES3.items():
        if P == 4 and size == "wide":
            continue  # no shape of its own: 16 elements are the widest tile
        CASES[f"euler3d-P{P}-{size}"] = (n, FAR, dict(order=P, dtType=1, CFL=0.4, uBound=0.4, pBound=1 / 1.4))
        CASES[f"ns3d-P{P}-{size}"] = (n, WALL3, dict(order=P, dtType=0, dt=1e-4, **NS))
CASES["advection3d-P3"] = ((7, 5, 4), {}, dict(order=3, equation=0, dtType=0, dt=1e-3))
CASES["advdiff3d-P2"] = ((7, 5, 4), {}, dict(order=2, equation=0, viscous=1, diffD=0.1, dtType=0, dt=1e-4))
CASES["penalty3d-P2"] = ((6, 5, 4), WALL3, dict(order=2, dtType=0, dt=1e-4, penFact=0.5, tau=0.1, **NS))
CASES["local-dt3d-P2"] = ((6, 5, 4), FAR, dict(order=2, dtType=2, CFL=0.3, uBound=0.4, pBound=1 / 1.4))
CASES["jameson3d-P2"] = ((6, 5, 4), {}, dict(order=2, dtType=1, CFL=0.3, timeType=5, pBound=1 / 1.4))
for P in (1, 2, 3, 4, 5):
    for n in ((53, 47), (9, 7)):  # 2491 = 78 x 32 - 5, and a mesh for the narrow tiles
        CASES[f"ns2d-P{P}-{n[0]}"] = (n, WALL3, dict(order=P, dtType=0, dt=1e-5, riemannType=P % 2, **NS))


def _state(pos, d, advection):
    x = pos
    w = [0.05 * np.prod(np.sin(2 * np.pi * x + 0.7 * k), -1) for k in range(5)]
    if advection:
        return (1 + w[0])[..., None]
    rho, v, p = 1 + w[0], [0.3 + w[1], w[2], w[3]][:d], (1 + w[4]) / 1.4
    return np.stack([rho, *(rho * q for q in v), p / 0.4 + 0.5 * rho * sum(q * q for q in v)], -1)


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("name", list(CASES))
def test_line_kernels_match_oracle(oracle, name, precision):
    from fr_learn_b200 import Solver, box2d, box3d

    n, bcs, kw = CASES[name]
    d = len(n)
    sides = {k: v for k, v in bcs.items() if d == 3 or not k.startswith("z")}
    mesh = box2d(*n, 0.0, 1.0, 0.0, 1.0, bcs=sides, perturb=0.1, seed=3) if d == 2 else \
        box3d(*n, (0.0,) * 3, (1.0,) * 3, bcs=sides, perturb=0.1, seed=3)
    oracle.lib().orc_set_threads(16)
    o = oracle.Oracle(oracle.params(nDims=d, **kw), mesh)
    g = Solver(mesh, precision=precision, **kw)
    U = _state(g.get("pos_spts"), d, kw.get("equation", 1) == 0)
    o.set("U_spts", U)
    g.set("U_spts", U)
    tol = 1e-12
    if precision == 0:
        o.calc_residual(0)
        g.calcResidual(0)
        assert relerr(g.get("divF_spts"), o.divF(0)) < tol
        assert relerr(g.getNormResidual(2), o.residual_norm(2)) < tol
    o.update(3)
    g.update(3)
    got, want = g.get("U_spts").ravel(), o.U().ravel()
    if precision == 0:
        assert relerr(got, want) < tol
        if kw["dtType"] == 1:
            assert abs(g.dt - o.dt) <= tol * o.dt
    else:
        assert np.linalg.norm(got - want) < 1e-6 * np.linalg.norm(want)
