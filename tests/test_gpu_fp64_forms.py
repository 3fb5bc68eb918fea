"""The FP64 residual kernels' reduced-instruction forms where their branches
lie - the entropy fix of the acoustic waves, operands outside the range of the
FP32 seeds, the ends of the limiter's screening - against the oracle."""
import numpy as np
import pytest

from oracle_lib import OracleSpace
from parity import assert_residual_close
from proteuscfd_gb300 import SolutionSpace, cases
from proteuscfd_gb300 import _native as N

pytestmark = pytest.mark.gpu


def random_states(kind, nrows, seed):
    """Rows of physical states: "sonic" around Mach 1 in random directions
    (the acoustic entropy fix switches on and off), "jumps" with densities and
    pressures over three decades."""
    rng = np.random.default_rng(seed)
    if kind == "sonic":
        rho, p = 1.4 * rng.uniform(0.8, 1.2, nrows), rng.uniform(0.8, 1.2, nrows)
        speed = np.sqrt(1.4 * p / rho) * rng.uniform(0.7, 1.3, nrows)
    else:
        rho, p = 10.0 ** rng.uniform(-2, 1, nrows), 10.0 ** rng.uniform(-2, 1, nrows)
        speed = np.sqrt(1.4 * p / rho) * rng.uniform(0.0, 3.0, nrows)
    d = rng.normal(size=(nrows, 3))
    u = d / np.linalg.norm(d, axis=1, keepdims=True) * speed[:, None]
    q = np.zeros((nrows, 10))
    q[:, 0], q[:, 1:4] = rho, rho[:, None] * u
    q[:, 4] = p / 0.4 + 0.5 * rho * speed ** 2
    return cases.with_aux(q)


@pytest.mark.parametrize("kind", ["sonic", "jumps"])
@pytest.mark.parametrize("dims", [(9, 7, 6), (2, 2, 2)])
def test_roe_flux_against_oracle(kind, dims):
    """First-order Roe fluxes of every edge and half-edge.  A component is
    formed with fewer than 200 roundings of terms no larger than 20 of its
    magnitude at Mach 3: 200 * 20 * 2^-53 = 4.4e-13, within the 1e-12 bar."""
    case = cases.euler_ramp(*dims, seed=4)
    m = cases.build_mesh(case)
    S = SolutionSpace(m, case.param)
    O = OracleSpace(m, case.param)
    q = random_states(kind, m.nnode + m.nbedge, 21)
    S.set_state(q)
    b, _ = S.compute_residuals()
    bo, _, kc = O.residual(q)
    assert kc == 0 and S.health()[0] == 0
    assert_residual_close(b, bo, O.last_babs)


@pytest.mark.parametrize("power", [-130, -40, 40, 120])
def test_roe_flux_scales_with_the_state(power):
    """The flux is linear in a common factor of density, momentum and energy.
    Factors of 2^-130 and 2^120 put every reciprocal and root outside the
    seeds' exponent range (2^-100 .. 2^100), so the plain operators run; a
    power of two changes no other rounding.  Same bound as above."""
    case = cases.euler_ramp(9, 7, 6, seed=4)
    m = cases.build_mesh(case)
    S = SolutionSpace(m, case.param)
    O = OracleSpace(m, case.param)
    q = random_states("jumps", m.nnode + m.nbedge, 22)
    S.set_state(q)
    b, _ = S.compute_residuals()
    O.residual(q)
    q[:, :5] *= 2.0 ** power
    S.set_state(cases.with_aux(q))
    bs, _ = S.compute_residuals()
    assert_residual_close(bs * 2.0 ** -power, b, O.last_babs)


@pytest.mark.parametrize("mach", [0.0, 0.3, 0.999, 1.6])
@pytest.mark.parametrize("noise", [0.0, 1e-9, 1e-3, 0.2])
def test_boundary_forms_against_oracle(mach, noise):
    """The far-field and slip-wall sub-iterations: flow into, out of, along
    and (exactly) not through the faces, sub- and supersonic, and phantom
    rows whose average with the node has no positive pressure; sub-iterations
    that reach their fixed point at once, after a few, or not.  Ten
    sub-iterations of about 50 roundings of terms up to 5 of the result:
    10 * 50 * 5 * 2^-53 = 2.8e-13, held to 1e-12 of the column's magnitude."""
    case = cases.euler_ramp(9, 7, 6, seed=4)
    p = case.param
    p.mach = mach
    p.bc_type = {1: N.BC_FARFIELD, 2: N.BC_FARFIELD, 3: N.BC_IMPERMEABLE_WALL, 4: N.BC_FARFIELD, 5: N.BC_SYMMETRY,
                 6: N.BC_FARFIELD}
    m = cases.build_mesh(case)
    S = SolutionSpace(m, p)
    O = OracleSpace(m, p)
    q = cases.perturbed_state(S.qinf(), m.nnode + m.nbedge, 5, amp=noise)
    if noise:
        rng = np.random.default_rng(6)
        far = np.flatnonzero(np.isin(m.bfactag, (1, 2, 4, 6)))
        q[m.nnode + rng.choice(far, len(far) // 8, replace=False), 4] *= -3.0
        q = cases.with_aux(q)
    S.set_state(q)
    S.update_bcs()
    qg, qo = S.get_state(), O.update_bcs(q)
    assert np.array_equal(np.isnan(qg), np.isnan(qo))
    scale = np.maximum(np.nanmax(np.abs(qo[:, :7]), axis=0), 1e-300)
    assert np.nanmax(np.abs(qg - qo)[:, :7] / scale) <= 1e-12


def limiter_state(kind, m, qinf, seed):
    """States that end in each branch of the limiter's FP32 screening: "flat"
    (every extrapolation leaves the value: no neighbour screens), "level"
    (noise of 1e-15: every neighbour ties within its bound), "noise" (one
    neighbour clears the others), "sheet" (equal values on two sides of a
    plane: neighbours tie at equal ratios), "small" and "large" (operands FP32
    cannot square)."""
    rng = np.random.default_rng(seed)
    n = m.nnode + m.nbedge
    q = np.tile(qinf, (n, 1))
    if kind == "sheet":
        q[:, :5] *= np.where(rng.uniform(size=n) < 0.5, 0.9, 1.1)[:, None]
    elif kind != "flat":
        amp = {"level": 1e-15, "noise": 0.01, "small": 0.01, "large": 0.01}[kind]
        q[:, :5] *= 1.0 + rng.uniform(-amp, amp, size=(n, 5))
        q[:, 3] = 0.0
    q[:, :5] *= {"small": 1e-19, "large": 1e19}.get(kind, 1.0)
    return cases.with_aux(q)


@pytest.mark.parametrize("kind", ["flat", "level", "noise", "sheet", "small", "large"])
@pytest.mark.parametrize("limiter", [1, 2, 3])
@pytest.mark.parametrize("dims", [(10, 8, 7), (3, 2, 2)])
def test_limiter_screening_against_oracle(kind, limiter, dims):
    """The limiter (with the pressure clip) of the GPU's own gradient: a value is one quotient of terms with fewer
    than 20 roundings, conditioned by at most 1e3 where the extrapolated
    change is above 1e-13 of the value: 20 * 1e3 * 2^-53 = 2.2e-12, held to
    1e-11 (the level field's own bound: its ratios hang on the last bits, so
    there only the range is checked)."""
    case = cases.ns_flatplate(*dims, seed=5)
    case.param.limiter = limiter
    m = cases.build_mesh(case)
    S = SolutionSpace(m, case.param)
    O = OracleSpace(m, case.param)
    q = limiter_state(kind, m, S.qinf(), 8)
    S.set_state(q)
    g = S.gradient()
    lg = S.limiter()
    if kind == "level":
        assert np.all((lg >= 0.0) & (lg <= 1.0))
        if limiter == 3:
            assert np.abs(lg - 1.0).max() <= 1e-9  # eps^2 outweighs 1e-15 noise
        return
    lo, _ = O.limiter(q, g)
    assert np.abs(lg - lo).max() <= 1e-11
