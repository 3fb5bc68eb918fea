"""The FP64 limiter's screening where its decisions are close: streams whose
variations are near the rounding of the values they sit on, and neighbours whose
ratios differ by about the screening bound - against the oracle."""
import numpy as np
import pytest

from oracle_lib import OracleSpace
from proteuscfd_gb300 import SolutionSpace, cases

pytestmark = pytest.mark.gpu


def near_tie_state(m, qinf, split, seed):
    """Two levels 10 % apart, as on either side of a sheet, each scattered by
    split: many neighbours of a node have ratios that differ by about split."""
    rng = np.random.default_rng(seed)
    n = m.nnode + m.nbedge
    q = np.tile(qinf, (n, 1))
    level = np.where(rng.uniform(size=n) < 0.5, 0.9, 1.1)[:, None]
    q[:, :5] *= level * (1.0 + rng.uniform(-split, split, size=(n, 5)))
    return cases.with_aux(q)


@pytest.mark.parametrize("state", [1e-16, 5e-16, 2e-15, 1e-13, 1e-11, 1e-9, 1e-8, "1e-7", "1e-6", "1e-5"])
@pytest.mark.parametrize("limiter", [1, 2, 3])
@pytest.mark.parametrize("dims", [(19, 14, 12), (3, 2, 2)])
def test_limiter_of_close_neighbours(state, limiter, dims):
    """A number is the amplitude of the stream's noise, a text the split of near
    ties.  grad.dx and the extrapolated value are rounded alike on both sides, so
    both take the same neighbour's ratio (or one within the other's rounding) and
    differ by the roundings of one value alone: fewer than 20 of terms no larger
    than twice the denominator, 20 * 2 * 2^-53 = 4.4e-15, held to 1e-14."""
    case = cases.ns_flatplate(*dims, seed=5)
    case.param.limiter = limiter
    m = cases.build_mesh(case)
    S = SolutionSpace(m, case.param)
    O = OracleSpace(m, case.param)
    if isinstance(state, str):
        q = near_tie_state(m, S.qinf(), float(state), 9)
    else:
        q = cases.perturbed_state(S.qinf(), m.nnode + m.nbedge, 9, amp=state)
    S.set_state(q)
    g = S.gradient()
    lg = S.limiter()
    lo, nclip = O.limiter(q, g)
    assert nclip == 0
    assert np.abs(lg - lo).max() <= 1e-14
