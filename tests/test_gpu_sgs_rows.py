"""The block Gauss-Seidel sweep that gives a lane a matrix row (six block rows
a warp), where its reads and its choice can go wrong: colours of fewer rows
than a warp takes, rows of no more and of far more blocks than its unrolled
part (20), colours on both sides of the FP64 size rule - against the oracle's
row update in the same colour order."""
import numpy as np
import pytest
from scipy.spatial import ConvexHull

from oracle_lib import OracleImplicit
from proteuscfd_gb300 import Mesh, Param, SolutionSpace, cases
from proteuscfd_gb300 import _native as N

pytestmark = pytest.mark.gpu


def stars(count, npts):
    """count separate balls of tets around a centre each, whose row has npts
    blocks."""
    k = np.arange(npts) + 0.5
    phi, th = np.arccos(1 - 2 * k / npts), np.pi * (1 + 5 ** 0.5) * k
    pts = np.c_[np.cos(th) * np.sin(phi), np.sin(th) * np.sin(phi), np.cos(phi)]
    tri = ConvexHull(pts).simplices
    inward = np.einsum("ij,ij->i", np.cross(pts[tri[:, 1]] - pts[tri[:, 0]], pts[tri[:, 2]] - pts[tri[:, 0]]),
                       pts[tri[:, 0]]) < 0
    tet = np.c_[np.zeros(len(tri), int), tri + 1]
    tet[inward] = tet[inward][:, [0, 1, 3, 2]]
    ball = np.vstack([[0.0, 0.0, 0.0], pts])
    at = [(npts + 1) * k for k in range(count)]
    xyz = np.vstack([ball + 3.0 * np.array([k % 30, k // 30, 0]) for k in range(count)])
    return Mesh.from_elements(xyz, np.vstack([tri + 1 + o for o in at]), np.ones(len(tri) * count, int),
                              np.vstack([tet + o for o in at]))


@pytest.mark.parametrize("prec", [0, 1], ids=["fp64", "fp32"])
@pytest.mark.parametrize("which", ["cell", "star21", "star40", "stars", "ragged"])
def test_sweeps_match_coloured_oracle(which, prec):
    """Three sweeps from zero.  A row sums at most 40 blocks of five products:
    FP64 200 * 2^-53 * 6 half sweeps' growth stays far within 1e-10 of the
    largest entry, FP32 200 * 2^-24 * 6 = 7e-5 within 2e-4."""
    if which in ("cell", "ragged"):
        c = cases.ns_flatplate(*((2, 2, 2) if which == "cell" else (37, 31, 23)), seed=3)
        m, prm = cases.build_mesh(c), c.param
    else:
        m = stars(900, 23) if which == "stars" else stars(1, int(which[4:]))
        prm = Param(gamma=1.4, mach=0.7, bc_type={1: N.BC_FARFIELD})
    S = SolutionSpace(m, prm)
    O = OracleImplicit(m, prm)
    S.set_state(cases.perturbed_state(S.qinf(), m.nnode + m.nbedge, 2))
    S.set_jacobian_precision(prec)
    S.compute_timesteps(5.0)
    S.compute_jacobians()
    cptr, rows = S.coloring()
    per_sm = np.diff(cptr).max() / 152
    assert (per_sm > 17) == (which in ("stars", "ragged")), per_sm
    b = np.random.default_rng(6).normal(size=(m.nnode, 5))
    Mlu, pv = O.lu(S.get_jacobian())
    xo = O.sgs_colored(Mlu, pv, b, 3, cptr, rows)
    x = S.sgs_rhs(b, 3, fp32=bool(prec))
    assert np.abs(x - xo).max() <= (2e-4 if prec else 1e-10) * np.abs(xo).max()
    S.close()
