"""Uploads are ordered before the kernels that read them.  A handle's stream is
created non-blocking, so its kernels do not wait for the legacy stream, on which
a copy from pageable memory may still be under way when cudaMemcpy returns: every
upload, and every clearing of device memory, is issued on the handle's own stream."""
import re
from pathlib import Path

import numpy as np
import pytest

from chem_cases import fr_states, mechanism
from proteuscfd_gb300.chem import ChemModel

CSRC = Path(__file__).resolve().parent.parent / "proteuscfd_gb300" / "csrc"


@pytest.mark.parametrize("source", ["chem.cu", "solver.cu"])
def test_no_upload_on_the_legacy_stream(source):
    text = (CSRC / source).read_text()
    assert "cudaStreamNonBlocking" in text
    uploads = [c for c in re.findall(r"cudaMemcpy\s*\([^;]*;", text) if "HostToDevice" in c]
    assert not uploads, uploads
    assert not re.findall(r"cudaMemset\s*\([^;]*;", text)


@pytest.mark.gpu
def test_every_handle_holds_the_same_mechanism():
    """The factors of Wilke's rule, which a kernel writes into the uploaded
    constants at creation, are in force in every handle: equal bits."""
    ref, rhoi, _, T = fr_states(64, seed=3)
    ref.viscosity = ref.density * ref.velocity
    ref.conductivity = ref.density * ref.velocity ** 3 / ref.temperature
    first = None
    for _ in range(40):
        C = ChemModel(mechanism())
        mu, k = C.transport(ref, rhoi, T)
        C.close()
        assert np.all(mu > 0.0) and np.all(np.isfinite(mu)) and np.all(k > 0.0) and np.all(np.isfinite(k))
        if first is None:
            first = mu, k
        assert np.array_equal(mu, first[0]) and np.array_equal(k, first[1])
