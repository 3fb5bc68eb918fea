"""States at the ends of FP64's range and states that are not finite: the results
are those of the plain forms, and a quantity formed from an infinite value does
not come out finite."""
import numpy as np
import pytest

from oracle_lib import OracleImplicit, OracleSpace
from proteuscfd_gb300 import SolutionSpace, cases
from proteuscfd_gb300 import _native as N

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("power", [-600, -150, 150, 600])
def test_wall_condition_scales_with_the_state(power):
    """The slip-wall sub-iterations are linear in a common factor of density,
    momentum and energy, and a power of two changes no rounding of theirs: within
    2.8e-13 of the column's magnitude as the boundary forms' test derives (ten
    sub-iterations of 50 roundings of terms up to 5 of the result), held to 1e-12."""
    case = cases.euler_ramp(9, 7, 6, seed=4)
    case.param.bc_type = {1: N.BC_SONIC_OUTFLOW, 2: N.BC_SONIC_OUTFLOW, 3: N.BC_IMPERMEABLE_WALL,
                          4: N.BC_IMPERMEABLE_WALL, 5: N.BC_SYMMETRY, 6: N.BC_SYMMETRY}
    m = cases.build_mesh(case)
    S = SolutionSpace(m, case.param)
    q = cases.perturbed_state(S.qinf(), m.nnode + m.nbedge, 5, amp=0.05)
    S.set_state(q)
    S.update_bcs()
    one = S.get_state()[:, :5]
    assert np.all(np.isfinite(one))
    q[:, :5] *= 2.0 ** power
    S.set_state(cases.with_aux(q))
    S.update_bcs()
    scaled = S.get_state()[:, :5] * 2.0 ** -power
    assert np.all(np.isfinite(scaled))
    assert (np.abs(scaled - one).max(axis=0) / np.abs(one).max(axis=0)).max() <= 1e-12
    S.close()


@pytest.mark.parametrize("value", [np.inf, -np.inf])
@pytest.mark.parametrize("component", [0, 1, 4])
def test_infinite_values_reach_time_step_and_residual(component, value):
    """A node with an infinite density, momentum or energy: the time steps and the
    momentum and energy residuals (those the viscous flux has) are NaN where the
    oracle's are, as a broken state shows itself."""
    case = cases.ns_flatplate(9, 8, 7, seed=5)
    case.param.sorder, case.param.limiter = 1, 0
    m = cases.build_mesh(case)
    S, O = SolutionSpace(m, case.param), OracleSpace(m, case.param)
    q = cases.perturbed_state(S.qinf(), m.nnode + m.nbedge, 5)
    q[(4 * 8 + 4) * 9 + 4, component] = value
    with np.errstate(invalid="ignore"):
        q = cases.with_aux(q)
    S.set_state(q)
    dt, _ = S.compute_timesteps(5.0)
    assert np.array_equal(np.isnan(dt), np.isnan(OracleImplicit(m, case.param).timestep(q, 5.0)[0]))
    g = S.gradient()
    b, _ = S.compute_residuals()
    bo, _, _ = O.residual(q, g)
    assert np.isnan(bo).any() and np.array_equal(np.isnan(b[:, 1:]), np.isnan(bo[:, 1:]))
    S.close()
