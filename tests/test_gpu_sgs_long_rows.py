"""The block Gauss-Seidel sweep with a lane per matrix row on rows longer than
its unrolled part of 20 blocks, as unstructured meshes have them, at the ends of
that part - against the oracle; and its equality with the FP64 kernel that small
meshes take."""
import numpy as np
import pytest
from scipy.spatial import ConvexHull

from oracle_lib import OracleImplicit
from proteuscfd_gb300 import Mesh, Param, SolutionSpace, cases
from proteuscfd_gb300 import _native as N

pytestmark = pytest.mark.gpu

SIZES = (19, 20, 21, 22, 39, 40, 41, 59, 60, 61, 79)


def ball(npts):
    """(points, triangles, tets) of a ball of tets around a centre whose row has
    npts blocks."""
    k = np.arange(npts) + 0.5
    phi, th = np.arccos(1 - 2 * k / npts), np.pi * (1 + 5 ** 0.5) * k
    pts = np.c_[np.cos(th) * np.sin(phi), np.sin(th) * np.sin(phi), np.cos(phi)]
    tri = ConvexHull(pts).simplices
    inward = np.einsum("ij,ij->i", np.cross(pts[tri[:, 1]] - pts[tri[:, 0]], pts[tri[:, 2]] - pts[tri[:, 0]]),
                       pts[tri[:, 0]]) < 0
    tri[inward] = tri[inward][:, [0, 2, 1]]
    return np.vstack([[0.0, 0.0, 0.0], pts]), tri + 1, np.c_[np.zeros(len(tri), int), tri + 1]


def balls(copies):
    """copies times a ball of every size, all around the origin: the copies are
    not connected, so their geometry, states and matrix rows have equal bits."""
    xyz, tris, tets, n = [], [], [], 0
    parts = [ball(s) for s in SIZES]
    for _ in range(copies):
        for p, t, e in parts:
            xyz.append(p)
            tris.append(t + n)
            tets.append(e + n)
            n += len(p)
    tris = np.vstack(tris)
    return Mesh.from_elements(np.vstack(xyz), tris, np.ones(len(tris), int), np.vstack(tets))


def solve(copies, prec):
    """(x of three sweeps, the oracle's, the first copy's blocks, rows of the
    largest colour)"""
    m = balls(copies)
    prm = Param(gamma=1.4, mach=0.7, bc_type={1: N.BC_FARFIELD})
    S, O = SolutionSpace(m, prm), OracleImplicit(m, prm)
    one = m.nnode // copies
    q = cases.perturbed_state(S.qinf(), one, 2)
    hb = cases.perturbed_state(S.qinf(), m.nbedge // copies, 3)
    S.set_state(np.vstack([np.tile(q, (copies, 1)), np.tile(hb, (copies, 1))]))
    S.set_jacobian_precision(prec)
    S.compute_timesteps(5.0)
    S.compute_jacobians()
    cptr, rows = S.coloring()
    A = S.get_jacobian()
    b = np.tile(np.random.default_rng(6).normal(size=(one, 5)), (copies, 1))
    x = S.sgs_rhs(b, 3, fp32=bool(prec))
    Mlu, pv = O.lu(A)
    xo = O.sgs_colored(Mlu, pv, b, 3, cptr, rows)
    first = A[:len(A) // copies].copy()
    S.close()
    return x, xo, first, np.diff(cptr).max()


@pytest.mark.parametrize("prec", [0, 1], ids=["fp64", "fp32"])
@pytest.mark.parametrize("copies", [1, 300])
def test_long_rows_against_oracle(copies, prec):
    """A row sums at most 79 blocks of five products over six half sweeps: FP64
    395 * 6 * 2^-53 far within 1e-10 of the largest entry, FP32 395 * 6 * 2^-24 =
    1.4e-4 within 2e-4."""
    x, xo, _, _ = solve(copies, prec)
    assert np.abs(x - xo).max() <= (2e-4 if prec else 1e-10) * np.abs(xo).max()


def test_fp64_kernels_give_equal_bits():
    """Few rows run the staged kernel, 300 copies of them (3,300 centres, more
    than 17 a multiprocessor) the lane-per-row kernel: the same sums in the same
    order, so each copy's x has the bits of the single one's."""
    x1, _, a1, _ = solve(1, 0)
    xn, _, an, rows = solve(300, 0)
    assert rows >= 17 * 152
    assert np.array_equal(a1, an)
    assert np.array_equal(xn.reshape(300, *x1.shape), np.broadcast_to(x1, (300, *x1.shape)))
