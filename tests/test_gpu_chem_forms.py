"""The reacting kernels' branches that the air mechanism does not reach -
temperature and concentration exponents of every code, pressure factors that
are no whole power - and both forms of the flux's per-record values, against
the oracle."""
import copy

import numpy as np
import pytest

from chem_cases import fr_edges, fr_records, fr_states, mechanism, states
from oracle_lib import OracleChemState, chem_rates
from proteuscfd_gb300.chem import ChemModel, model_struct

pytestmark = pytest.mark.gpu


def variant(n, rtype, stoich):
    """The air mechanism with every reaction's temperature exponent and form
    replaced, and with stoich the first reaction's exponents (nu, whole or not)."""
    spec = copy.deepcopy(mechanism())
    for r in spec["reactions"]:
        r["n"], r["type"] = n, rtype
        if rtype in (0, 1):
            r["EA"] *= 8.314
    r = spec["reactions"][0]
    r["nup"][0], r["nupp"][1] = stoich
    return spec


@pytest.mark.parametrize("n", [0.0, 1.0, -1.0, 0.5, -1.5, 4.0, -4.0, 4.5, 0.37])
@pytest.mark.parametrize("rtype,stoich", [(2, (1.0, 2.0)), (1, (0.5, 3.0)), (0, (1.0, 1.0)), (3, (2.0, 0.0)),
                                          (2, (1.0, 4.0))])
def test_rate_exponent_codes(n, rtype, stoich):
    """Rates and source Jacobian.  A rate constant is an exponential of an
    argument up to 300 in size: 300 * 4 * 2^-53 = 1.3e-13 relative, the
    reactions' sums a few of it: 1e-12 of the node's largest rate; the
    differences divide by 1e-8: 1e-5 of the column's largest entry and the
    largest source, as in the Jacobian's parity test."""
    spec = variant(n, rtype, stoich)
    rho, T = states(300, seed=7)
    T = np.clip(T, 800.0, None)
    C = ChemModel(spec)
    m = model_struct(spec)
    w, wo = C.production_rates(rho, T), chem_rates(m, rho, T)
    scale = np.abs(wo).max(axis=1, keepdims=True)
    assert (np.abs(w - wo) / np.where(scale > 0, scale, 1.0)).max() < 1e-12
    ref, frho, fvel, fT = fr_states(130, seed=9)
    fT = np.clip(fT, 1500.0 / ref.temperature, None)
    q = fr_records(ref, frho, fvel, fT)
    vol = np.linspace(0.5, 2.0, len(fT))
    A, Ao = C.source_jacobian(ref, 2.5e-4, q, vol), OracleChemState(m, ref).source_jacobian(q, vol, 2.5e-4)
    src = chem_rates(m, (q[:, :5] * ref.density).copy(), q[:, 8] * ref.temperature)
    smax = np.abs(vol[:, None] * src / (ref.density / 2.5e-4)).max(axis=1)
    scale = np.abs(Ao).max(axis=1) + smax[:, None]
    assert (np.abs(A - Ao) / np.where(scale > 0, scale, 1.0)[:, None, :]).max() < 1e-5
    C.close()


@pytest.mark.parametrize("nedge", [1, 99, 100, 101, 1000])
def test_hllc_per_record_values(nedge):
    """200 records: up to 100 edges the faces form their records' speed of
    sound and enthalpy themselves, beyond they read them; the values and the
    bar are those of the flux parity test (1e-12 of the face's terms)."""
    ref, rhoi, vel, T = fr_states(200, seed=5)
    q = fr_records(ref, rhoi, vel, T)
    edges, avec = fr_edges(200, nedge, seed=6)
    C = ChemModel(mechanism())
    o = ChemModel.flux_opts(1.0, 0.0)
    f = C.hllc_flux(ref, o, q, edges, avec)
    fo, bad = OracleChemState(model_struct(mechanism()), ref).hllc_batch(o, q, edges, avec)
    assert bad == 0
    assert (np.abs(f - fo) / np.abs(fo).max(axis=1, keepdims=True)).max() < 1e-12
    C.close()
