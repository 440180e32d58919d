"""One handle used for many gradients: captured segment graphs and stage slots are
kept between runs, so every gradient is compared with a fresh handle's.  dJ/dU_0 to
the bit; dJ/dtheta is summed by atomics, so to rounding (1e-12 of it)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

NS = dict(viscous=1, mu_inf=0.05, prandtl=0.72, penFact=0.3, TWall=1.0, RGas=1 / 1.4)
THETA = np.array([0.1, 1.0, 0.2, 0.0, 0.3])


def _solver(visc):
    from fr_learn_b200 import Solver, bump2d

    kw = dict(order=2, riemannType=1, uBound=0.5, pBound=1.0, dtType=0, dt=1e-3)
    if visc:
        kw.update(NS)
    return Solver(bump2d(6, 3, **(dict(bc_wall="adiabatic_noslip") if visc else {})), **kw)


def _gradient(s, k, nsteps, every, variant=None):
    if variant is not None:
        s.set_tile_variant(variant)
    s.setInitialCondition(0)
    U = s.get("U_spts")
    s.set("U_spts", U * (1 + 0.01 * np.random.default_rng(k).standard_normal(U.shape)))
    s.adjoint_forward(nsteps, every)
    s.objective("entropy")
    return s.adjoint_backward(None, THETA)


@pytest.mark.parametrize("visc", [False, True])
def test_gradients_of_one_handle_equal_a_fresh_handles(visc):
    """New states, other lengths and intervals (slots reused, grown, a second set
    added), every stage kept, and a change of tile shape, which drops the graphs."""
    one = _solver(visc)
    runs = [(7, 3, None), (7, 3, None), (7, 2, None), (12, 5, None), (8, 0, None), (7, 3, None), (3, 3, None)]
    if not visc:
        runs += [(7, 3, 5), (7, 3, 10), (9, 4, 0)]
    for k, (nsteps, every, variant) in enumerate(runs):
        lam, th = _gradient(one, k, nsteps, every, variant)
        want, th0 = _gradient(_solver(visc), k, nsteps, every, variant)
        assert np.array_equal(lam, want), (k, nsteps, every)
        assert abs(th - th0) <= 1e-12 * abs(th0), (k, th, th0)
        # other calls on the handle between gradients
        one.update(3)
        one.calcResidual(0)
