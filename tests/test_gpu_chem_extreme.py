"""The reacting kernels beside values that are not finite: what the plain forms
give."""
import numpy as np
import pytest

from chem_cases import fr_records, fr_states, mechanism, states
from oracle_lib import OracleChemState, chem_rates
from proteuscfd_gb300 import Mesh
from proteuscfd_gb300.chem import ChemModel, model_struct

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("value", [np.inf, -np.inf])
@pytest.mark.parametrize("chi", [0.0, 0.5])
def test_limiter_beside_infinite_values(chi, value):
    """One node's density, velocity, temperature or pressure infinite, with the
    gradient that follows: away from the node itself, whose values are broken, the
    limiter agrees with the oracle's within the parity test's 1e-12 and is NaN
    nowhere else."""
    m = Mesh.box(9, 8, 7, jitter=0.2, seed=10)
    ref, rhoi, vel, T = fr_states(m.nnode + m.nbedge, seed=27)
    base = fr_records(ref, rhoi, vel, T)
    C, O = ChemModel(mechanism()), OracleChemState(model_struct(mechanism()), ref)
    C.attach_mesh(m)
    i = (4 * 8 + 4) * 9 + 4
    for component in (0, 3, 5, 8, 9):
        q = base.copy()
        q[i, component] = value
        g = C.gradient(q)
        lim, lo = C.limiter(chi, q, g), O.limiter(m, q, g, chi)
        others = np.arange(m.nnode) != i
        with np.errstate(invalid="ignore"):
            assert np.array_equal(np.isnan(lim[others]), np.isnan(lo[others])), component
            assert np.nanmax(np.abs(lim - lo)[others]) <= 1e-12
    C.close()


@pytest.mark.parametrize("value", [np.inf, -np.inf])
@pytest.mark.parametrize("species", range(5))
def test_rates_of_infinite_densities(species, value):
    """Infinite rates are infinite and NaN ones NaN where the oracle's are."""
    rho, T = states(300, seed=7)
    rho[::7, species] = value
    C = ChemModel(mechanism())
    w, wo = C.production_rates(rho, T), chem_rates(model_struct(mechanism()), rho, T)
    assert np.array_equal(np.isnan(w), np.isnan(wo))
    assert np.array_equal(w[np.isinf(wo)], wo[np.isinf(wo)]) and np.array_equal(np.isinf(w), np.isinf(wo))
    C.close()
