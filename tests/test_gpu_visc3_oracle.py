"""3D viscous updates against the oracle: state, traces of the state and dt, over
periodic, walled (LDG penalty), advection-diffusion and Sutherland cases.  FP64 to
rounding (1e-12), the mixed mode to 1e-6 in the 2-norm."""
import numpy as np
import pytest

from conftest import relerr
from test_gpu_parity import _visc3_cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("case", list(_visc3_cases()))
def test_visc3_update_matches_oracle(oracle, precision, case):
    from fr_learn_b200 import Solver

    mesh, ic, a0, kw = _visc3_cases()[case]
    o = oracle.Oracle(oracle.params(nDims=3, **kw), mesh)
    o.set_ic(ic, a0)
    g = Solver(mesh, precision=precision, **kw)
    g.setInitialCondition(ic, a0)
    o.update(5)
    g.update(5)
    if kw["dtType"] == 1:
        assert abs(g.dt - o.dt) <= (1e-12 if precision == 0 else 1e-6) * o.dt
    oracle.lib().orc_extrapolate_u(o.h)
    for name in ("U_spts", "U_fpts"):
        got, want = g.get(name).ravel(), o.get(name)
        if precision == 0:
            assert relerr(got, want) < 1e-12, name
        else:
            assert np.linalg.norm(got - want) < 1e-6 * np.linalg.norm(want), name
