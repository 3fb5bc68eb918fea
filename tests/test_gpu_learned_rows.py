"""The learned preconditioner's kernels at the sizes where their row pairs,
tiles and node runs end: fewer nodes than a half-warp row pair per warp, rows
of more than 16 and more than 32 neighbours, the last size with 64-row blocks
and one with 128-row blocks - forward pass and gradient against the oracle."""
import numpy as np
import pytest

from oracle_lib import OracleNet, lp_random_params
from proteuscfd_gb300 import Param, SolutionSpace, cases
from proteuscfd_gb300 import _native as N
from test_gpu_learned import FWD_RTOL, GRAD_RTOL, rel
from test_gpu_sgs_rows import stars

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("which", [(2, 2, 2), (5, 5, 5), (9, 8, 7), "star17", "star70", "stars", (38, 32, 32),
                                   (43, 31, 30)], ids=str)
def test_forward_and_gradient(which):
    """Outputs and gradients differ from the oracle's by flips of BF16
    roundings (2^-8 each) alone, whatever the sizes: the bars of the parity
    tests on ordinary meshes hold."""
    if isinstance(which, str):
        m = stars(60, 33) if which == "stars" else stars(1, int(which[4:]))
        prm = Param(gamma=1.4, mach=0.7, bc_type={1: N.BC_FARFIELD})
    else:
        c = cases.ns_flatplate(*which, seed=3)
        m, prm = cases.build_mesh(c), c.param
    S = SolutionSpace(m, prm)
    S.set_state(cases.perturbed_state(S.qinf(), m.nnode + m.nbedge, 1))
    S.lp_init(3)
    net = OracleNet(m)
    rng = np.random.default_rng(5)
    x = rng.uniform(-1, 1, (m.nnode, N.LP_NIN)).astype(np.float32)
    t = rng.uniform(-1, 1, (m.nnode, 5)).astype(np.float32)
    w = lp_random_params(9)
    S.lp_set_params(w)
    assert rel(S.lp_forward(x), net.forward(x, w, emulate=1)) < FWD_RTOL
    loss, g = S.lp_loss_grad(x, t)
    loss_ref, g_ref = net.loss_grad(x, t, w, emulate=1)
    assert abs(loss - loss_ref) <= 1e-3 * loss_ref
    cuts = [0, 704, 768] + [768 + l * 8576 + o for l in range(3) for o in (256, 320, 4416, 8512, 8576)] + [26816, 26821]
    for a, e in zip(cuts, cuts[1:]):
        assert rel(g[a:e], g_ref[a:e]) < GRAD_RTOL, (a, rel(g[a:e], g_ref[a:e]))
    S.close()
