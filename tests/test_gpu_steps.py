"""Runs of steps in one graph, and the host-buffer call's small-state path: the
same bits as the steps one by one."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _cases():
    from fr_learn_b200 import box2d, box3d

    ns = dict(viscous=1, mu_inf=0.01, prandtl=0.72, uBound=0.2, pBound=1 / 1.4, TWall=1.0, RGas=1 / 1.4)
    walls = dict(ymin="isothermal_noslip", ymax="isothermal_noslip")
    return {
        "vortex-cfl-rusanov": (box2d(9, 8, -10, 10, -10, 10, perturb=0.1, seed=1), 1, dict(order=3, dtType=1, CFL=0.4)),
        "vortex-cfl-roe-mixed": (box2d(33, 31, -10, 10, -10, 10, perturb=0.1, seed=2), 1,
                                 dict(order=4, riemannType=1, dtType=1, CFL=0.4, precision=1)),
        "advection-fixed": (box2d(8, 7), 0, dict(order=2, equation=0, dtType=0, dt=1e-3)),
        "jameson-cfl": (box2d(6, 7, -10, 10, -10, 10), 1, dict(order=2, dtType=1, CFL=0.3, timeType=5)),
        "local-dt": (box2d(6, 7, -10, 10, -10, 10), 1, dict(order=2, dtType=2, CFL=0.3)),
        "rk2-cfl": (box2d(6, 7, -10, 10, -10, 10), 1, dict(order=2, dtType=1, CFL=0.2, timeType=2)),
        "euler3d-cfl": (box3d(4, 3, 5, perturb=0.1, seed=3), 10, dict(order=2, dtType=1, CFL=0.3)),
        "ns2d-walls-cfl": (box2d(7, 6, -1, 1, -1, 1, bcs=walls), 0, dict(order=2, dtType=1, CFL=0.05, **ns)),
    }


CASES = ["vortex-cfl-rusanov", "vortex-cfl-roe-mixed", "advection-fixed", "jameson-cfl", "local-dt", "rk2-cfl",
         "euler3d-cfl", "ns2d-walls-cfl"]


def _same(a, b):
    assert np.array_equal(a.get("U_spts"), b.get("U_spts"))
    assert a.time == b.time and a.dt == b.dt and a.iter == b.iter


@pytest.mark.parametrize("name", CASES)
def test_runs_of_steps_equal_single_steps(name):
    """64 steps are taken one by one before runs begin: 64 + 3 runs + 5 left, then
    a call of 7 (no run) and one of 8; the same with a residual monitor."""
    from fr_learn_b200 import Solver

    mesh, ic, kw = _cases()[name]
    for monitor in (False, True):
        a, b = Solver(mesh, **kw), Solver(mesh, **kw)
        for s in (a, b):
            s.setInitialCondition(ic, 0.2)
            s.setMonitor(monitor)
        for n in (93, 7, 8):
            a.update(n)
            for _ in range(n):
                b.update(1)
            _same(a, b)
            if monitor:
                assert np.array_equal(a.getNormResidual(2), b.getNormResidual(2))


def test_run_stops_at_the_step_that_recomputes_the_wave_speeds():
    from fr_learn_b200 import Solver

    mesh, ic, kw = _cases()["vortex-cfl-rusanov"]
    a, b = Solver(mesh, **kw), Solver(mesh, **kw)
    for s in (a, b):
        s.setInitialCondition(ic)
        s.update(70)
        s.setIter(0, 10)  # step 11 is the first of a run: wave speeds and dt anew
    a.update(40)
    for _ in range(40):
        b.update(1)
    _same(a, b)


@pytest.mark.parametrize("side", [8, 40])  # below and above the size that is written to the host directly
@pytest.mark.parametrize("pinned", [False, True])
def test_host_buffer_call_equals_device_steps(side, pinned):
    import torch
    from fr_learn_b200 import Solver, box2d

    mesh = box2d(side, 9, -10, 10, -10, 10, perturb=0.1, seed=4)
    kw = dict(order=4, riemannType=1, dtType=1, CFL=0.4)
    a, b = Solver(mesh, **kw), Solver(mesh, **kw)
    b.setInitialCondition(1)
    U = torch.empty((b.nSpts, b.nEles, b.nFields), dtype=torch.float64, pin_memory=pinned)
    U.numpy()[...] = b.get("U_spts")
    for n in (1, 2, 9):
        a.update_host(U.numpy(), n)
        b.update(n)
        assert np.array_equal(U.numpy(), b.get("U_spts"))
        assert a.dt == b.dt and a.time == b.time
