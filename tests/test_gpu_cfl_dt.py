"""What a caller sees of the CFL dt where a step's last stage computes the next
step's: 3D and viscous runs and the 2D line kernels.  The reference's params->dt is
the dt of the step just taken until the next calcDt (src/solver.cpp:212-250,
:293-305), and it is that dt that writeResidual checks (src/output.cpp:823-841)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ERR_NAN, ERR_DT = 3, 5
NS = dict(viscous=1, mu_inf=0.01, prandtl=0.72, uBound=0.2, pBound=1 / 1.4, TWall=1.0, RGas=1 / 1.4)
NAMES = ["euler3d", "euler3d-mixed", "ns3d", "ns2d", "euler2d-line"]


def _make(name, monkeypatch, **extra):
    from fr_learn_b200 import Solver, box2d, box3d

    mesh, ic, kw = {
        "euler3d": (box3d(4, 3, 5, perturb=0.1, seed=3), 10, dict(order=2)),
        "euler3d-mixed": (box3d(4, 3, 5, perturb=0.1, seed=3), 10, dict(order=2, precision=1)),
        "ns3d": (box3d(3, 3, 4, (0, 0, 0), (6.28,) * 3, perturb=0.05, seed=3), 10, dict(order=3, **NS)),
        "ns2d": (box2d(7, 6, -5, 5, -5, 5, perturb=0.1, seed=5), 1, dict(order=3, **NS)),
        "euler2d-line": (box2d(9, 7, -10, 10, -10, 10, perturb=0.1, seed=1), 1, dict(order=3)),
    }[name]
    if name == "euler2d-line":
        monkeypatch.setenv("FRG_KERNEL", "generic")
    s = Solver(mesh, dtType=1, **kw, **extra)
    s.setInitialCondition(ic, 0.2)
    return s


@pytest.mark.parametrize("name", NAMES)
def test_dt_error_belongs_to_the_step_that_used_it(monkeypatch, name):
    """Runs far beyond the stable CFL number: a step fails with the dt error exactly
    when the dt it used is below 1e-13 or a NaN, and otherwise with the NaN error."""
    from fr_learn_b200 import FrgError

    seen = set()
    for cfl in (3.0, 30.0, 100.0, 1e3, 1e5):
        s = _make(name, monkeypatch, CFL=cfl)
        errors = 0
        for _ in range(60):
            code = 0
            try:
                s.update(1)
            except FrgError as e:
                code = e.code
            dt = s.dt
            assert (code == ERR_DT) == (not dt >= 1e-13), (cfl, s.iter, code, dt)
            if code != ERR_DT:
                U = s.get("U_spts")  # the check reads the density and the energy
                assert (code == ERR_NAN) == bool(np.isnan(U[..., [0, -1]]).any()), (cfl, s.iter, code)
            seen.add(code)
            errors += code != 0
            if errors == 3:
                break
    assert len(seen) > 1  # the runs did blow up


@pytest.mark.parametrize("name", NAMES)
def test_element_dt_and_manual_stage_are_the_last_steps(monkeypatch, name):
    """The smallest of the elements' dt is the dt that frg_get_time gives, and a
    stage taken by hand uses it, after single steps, several and a run of steps."""
    s = _make(name, monkeypatch, CFL=0.1)
    for n in (1, 3, 80, 2):
        s.update(n)
        dt = s.dt
        assert abs(s.get("ele_dt").min() - dt) <= 1e-14 * dt, n
    s.copyUspts_U0()
    U0 = s.get("U_spts")
    s.calcResidual(0)
    s.timeStepA(0, 0.5)
    d = s.get("divF_spts", 0) / s.get("detJac_spts")[..., None]
    used = float(((U0 - s.get("U_spts")) * d).sum() / (0.5 * (d * d).sum()))
    # a difference of two states: rounding of the state over the step's change
    assert abs(used - dt) <= 1e-9 * dt
