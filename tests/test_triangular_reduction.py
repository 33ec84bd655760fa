"""The triangular shared-memory reduction of complex matrices (automatic for orders 175 to 230) and the
register-resident one at its largest orders (177 to 192, real): mixed energies against the oracle at the
mixed bar of 1e-6 eV. 178 and 226 leave a ragged last row tile, 181 and 229 one short strip; the batch of
320 gives every SM more than one matrix, so that a CTA's second matrix reuses its shared memory."""
import numpy as np
import pytest

from ultimateepm_gb300 import _native as N
from ultimateepm_gb300 import api

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("key,shells,nl,soc", [("GaAs", 8, True, True), ("GaAs", 12, True, False), ("GaAs", 9, True, True),
                                               ("InAs", 13, True, False), ("Ge", 12, True, False)])
def test_automatic_reductions_near_their_limits(gpu, oracle, mats, key, shells, nl, soc):
    G = oracle.generate_basis(shells)
    ks = oracle.sample_first_bz(4, 21)
    ctx = api._Context(api.Material(key, raw=N.UepmMaterial.from_buffer_copy(bytes(mats[key]))), G, nl, soc, N.UEPM_PREC_MIXED)
    E, _, _, st = ctx.solve(np.tile(ks, (80, 1)), 10)
    ctx.close()
    ref = oracle.band_structure(mats[key], G, ks, 10, nl=nl, soc=soc)["E"]
    assert not st.any()
    assert np.abs(E[:4] - ref).max() <= 1e-6
    assert np.array_equal(E, np.tile(E[:4], (80, 1)))
