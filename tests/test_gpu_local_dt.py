"""Local time steps (dtType 2): the state, the time and dt of every kernel that a
step can take.  The reference's time advances by params->dt, which calcDt leaves as
the smallest element's (src/solver.cpp:293-305).

Tolerance: FP64 agrees with the reference's algorithm to rounding (1e-12)."""
import numpy as np
import pytest

from conftest import relerr

pytestmark = pytest.mark.gpu

NS = dict(viscous=1, mu_inf=0.01, prandtl=0.72, uBound=0.2, pBound=1 / 1.4, TWall=1.0, RGas=1 / 1.4)


def _cases():
    from fr_learn_b200 import box2d, box3d

    return {
        "euler2d": (box2d(9, 7, -10, 10, -10, 10, perturb=0.1, seed=1), 1, dict(order=3, riemannType=1)),
        "euler3d": (box3d(4, 3, 5, perturb=0.1, seed=3), 10, dict(order=2)),
        "ns2d": (box2d(7, 6, -5, 5, -5, 5, perturb=0.1, seed=5), 1, dict(order=2, **NS)),
        "ns3d": (box3d(3, 3, 4, (0, 0, 0), (6.28,) * 3, perturb=0.05, seed=6), 10, dict(order=2, **NS)),
    }


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("name", ["euler2d", "euler3d", "ns2d", "ns3d"])
def test_local_dt_state_and_time(oracle, monkeypatch, name, precision):
    from fr_learn_b200 import Solver

    mesh, ic, kw = _cases()[name]
    kw = dict(kw, dtType=2, CFL=0.2)
    o = oracle.Oracle(oracle.params(nDims=mesh.nDims, **kw), mesh)
    o.set_ic(ic, 0.2)
    o.update(3)
    solvers = [(v, Solver(mesh, precision=precision, **kw)) for v in range(12 if name == "euler2d" else 1)]
    monkeypatch.setenv("FRG_KERNEL", "generic")
    solvers.append(("line", Solver(mesh, precision=precision, **kw)))
    first = None
    for v, s in solvers:
        if v != "line" and s.tile_variant_count() > 1:
            s.set_tile_variant(v)
        s.setInitialCondition(ic, 0.2)
        s.update(3)
        got, want = s.get("U_spts"), o.U()
        if precision == 0:
            assert relerr(got, want) < 1e-12, v
            assert abs(s.time - o.time) <= 1e-12 * o.time, (v, s.time, o.time)
            assert abs(s.dt - o.dt) <= 1e-12 * o.dt, v
        else:
            # the wave speeds that dt comes from are FP32's: 1e-6, as the state
            assert np.linalg.norm(got - want) < 1e-6 * np.linalg.norm(want), v
            assert abs(s.time - o.time) <= 1e-6 * o.time, (v, s.time, o.time)
        if v != "line":  # the tile shapes agree to the bit
            first = first or (got, s.time)
            assert np.array_equal(got, first[0]) and s.time == first[1], v
