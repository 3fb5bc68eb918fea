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


def limiter_restated(m, q, g, vol, node, eq):
    """Kernel_VenkatMod's minimum of one node and equation as the limiter keeps it:
    a fraction compared by cross-multiplication, neighbours in edge order."""
    e = np.asarray(m.edges)
    qi = q[node, eq]
    ends = [(k, e[k, 1] if e[k, 0] == node else e[k, 0]) for k in np.flatnonzero((e == node).any(axis=1))]
    hi, lo = 0.0, 0.0
    for _, j in ends:
        hi, lo = (hi if hi > q[j, eq] else q[j, eq]), (lo if lo < q[j, eq] else q[j, eq])
    ep2 = 6.0 * np.pi * vol[node]
    n, d = np.float64(1.0), np.float64(1.0)
    for _, j in ends:
        dx = 0.5 * (m.xyz[j] - m.xyz[node])
        Q = qi + ((g[node, 3 * eq] * dx[0] + g[node, 3 * eq + 1] * dx[1]) + g[node, 3 * eq + 2] * dx[2])
        DM, DP = Q - qi, (hi if Q > qi else lo) - qi
        num, den = DP * DP + ep2 + 2.0 * DM * DP, DP * DP + ep2 + DM * (DP + 2.0 * DM)
        if num * d < n * den:
            n, d = num, den
    v = n if d == 1.0 else n / d
    return 0.0 if v < 0.0 else v


@pytest.mark.parametrize("value", [np.inf, -np.inf, 1e200])
@pytest.mark.parametrize("component", [0, 1, 4])
def test_limiter_beside_infinite_values(component, value):
    """Nodes with an infinite or overflowing neighbour or gradient: the limiter's
    raw values before the pressure clip (which zeroes a node's five values) are
    the restatement's, NaN where it is, else within the limiter test's 1e-11."""
    case = cases.ns_flatplate(9, 8, 7, seed=5)
    m = cases.build_mesh(case)
    S = SolutionSpace(m, case.param)
    q = cases.perturbed_state(S.qinf(), m.nnode + m.nbedge, 5)
    i = (4 * 8 + 4) * 9 + 4
    q[i, component] = value
    with np.errstate(all="ignore"):
        q = cases.with_aux(q)
        S.set_state(q)
        g, lim = S.gradient(), S.limiter()
        e = np.asarray(m.edges)
        near = sorted(set(e[(e == i).any(axis=1)].ravel()))
        seen = 0
        for node in near:
            if np.all(lim[node] == 0.0):
                continue
            for eq in range(5):
                r = limiter_restated(m, q, g, m.vol, node, eq)
                assert np.isnan(r) == np.isnan(lim[node, eq]), (node, eq, r, lim[node, eq])
                assert np.isnan(r) or abs(r - lim[node, eq]) <= 1e-11
                seen += 1
    assert seen
    S.close()
