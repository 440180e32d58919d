"""Ensemble mode on the line kernels (3D, viscous): cases of one handle with their
own CFL dt give what each case gives alone.

Tolerance: the union's mesh may take another block shape than a case alone, so the
two agree to rounding: 1e-12 in FP64; in the mixed mode FP32 stage states round, and
both are held to 1e-6 in the 2-norm, as every parity test."""
import numpy as np
import pytest

from conftest import relerr

pytestmark = pytest.mark.gpu

NS = dict(viscous=1, mu_inf=0.01, prandtl=0.72, uBound=0.2, pBound=1 / 1.4, TWall=1.0, RGas=1 / 1.4)


def _cases(d):
    from fr_learn_b200 import box2d, box3d

    if d == 2:
        return [box2d(4, 3, -5, 5, -5, 5, perturb=0.1, seed=1), box2d(5, 6, -2, 3, -2, 3, perturb=0.1, seed=2)]
    return [box3d(3, 4, 3, (0, 0, 0), (1, 1, 1), perturb=0.1, seed=1),
            box3d(5, 3, 4, (0, 0, 0), (3, 2, 2), perturb=0.1, seed=2)]


def _state(pos, k, d):
    w = [0.05 * np.prod(np.sin(1.3 * pos + 0.7 * q + k), -1) for q in range(5)]
    rho, v, p = 1 + w[0], [0.3 + k + w[1], w[2], w[3]][:d], (1 + w[4]) / 1.4
    return np.stack([rho, *(rho * q for q in v), p / 0.4 + 0.5 * rho * sum(q * q for q in v)], -1)


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("d, visc", [(3, 0), (3, 1), (2, 1)])
def test_grouped_cfl_cases_equal_cases_alone(d, visc, precision):
    from fr_learn_b200 import Solver, concat_meshes

    cases = _cases(d)
    union, grp = concat_meshes(cases)
    kw = dict(order=2, dtType=1, CFL=0.1, precision=precision, **(NS if visc else dict(pBound=1 / 1.4)))
    e = Solver(union, **kw)
    e.set_groups(grp, 2)
    pos = e.get("pos_spts")
    e.set("U_spts", np.concatenate([_state(pos[:, grp == k], k, d) for k in range(2)], axis=1))
    alone = []
    for k, m in enumerate(cases):
        s = Solver(m, **kw)
        s.set("U_spts", _state(s.get("pos_spts"), k, d))
        alone.append(s)
    for n in (1, 5, 80):  # single steps, then runs of steps
        e.update(n)
        U, (t, dt) = e.get("U_spts"), e.group_times()
        for k, s in enumerate(alone):
            s.update(n)
            got, want = U[:, grp == k], s.get("U_spts")
            if precision == 0:
                assert relerr(got, want) < 1e-12, (n, k)
                assert abs(t[k] - s.time) <= 1e-12 * s.time and abs(dt[k] - s.dt) <= 1e-12 * s.dt, (n, k)
            else:
                assert np.linalg.norm(got - want) < 1e-6 * np.linalg.norm(want), (n, k)
                assert abs(t[k] - s.time) <= 1e-6 * s.time and abs(dt[k] - s.dt) <= 1e-6 * s.dt, (n, k)


@pytest.mark.parametrize("visc", [0, 1])
def test_grouped_dt_error_belongs_to_the_step_that_used_it(visc):
    """A group whose dt falls below 1e-13 raises the dt error in the step that uses
    it; the other group's dt is fine throughout."""
    from fr_learn_b200 import FrgError, Solver, concat_meshes

    cases = _cases(3)
    union, grp = concat_meshes(cases)
    kw = dict(order=2, dtType=1, CFL=30.0, **(NS if visc else dict(pBound=1 / 1.4)))
    e = Solver(union, **kw)
    e.set_groups(grp, 2)
    pos = e.get("pos_spts")
    e.set("U_spts", np.concatenate([_state(pos[:, grp == k], k, 3) for k in range(2)], axis=1))
    failed = 0
    for _ in range(60):
        code = 0
        try:
            e.update(1)
        except FrgError as err:
            code = err.code
        dt = e.group_times()[1]
        assert (code == 5) == (not (dt >= 1e-13).all()), (code, dt)
        failed += code != 0
        if failed == 2:
            break
    assert failed
