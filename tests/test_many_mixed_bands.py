"""Mixed solves with the most bands, 33 to 36: the projected pencil is of order 37 to 40, in quaternion form of whole
pairs (34 bands and their guards make 38, 35 make 40), and the small solver's two matrices per block then exceed the
shared memory for complex matrices."""
import numpy as np
import pytest

import fake_runtime
from ultimateepm_gb300 import _native as N
from ultimateepm_gb300 import api

KINDS = [("Ge", True, True), ("GaAs", True, True), ("InP", True, False), ("Ge", True, False)]


@pytest.mark.parametrize("key,nl,soc", KINDS)
def test_every_number_of_bands_is_launched(native, tmp_path, key, nl, soc):
    cases = [dict(material=key, shells=6, nl=nl, soc=soc, mixed=True, bands=nb, k=3) for nb in (33, 34, 35, 36)]
    assert [error for error, _, _ in fake_runtime.run(tmp_path, *cases)] == [None] * 4


@pytest.mark.gpu
@pytest.mark.parametrize("nb", [34, 35, 36])
@pytest.mark.parametrize("key,nl,soc", KINDS)
def test_against_the_oracle(gpu, oracle, mats, key, nl, soc, nb):
    """Energies within the mixed bar of 1e-6 eV, vectors orthonormal to 1e-8, an odd number of matrices."""
    G, ks = oracle.generate_basis(7), oracle.sample_first_bz(5, 3)
    ctx = api._Context(api.Material(key, raw=N.UepmMaterial.from_buffer_copy(bytes(mats[key]))), G, nl, soc, N.UEPM_PREC_MIXED)
    E, X, _, st = ctx.solve(ks, nb, vectors=True)
    ctx.close()
    ref = oracle.band_structure(mats[key], G, ks, nb, nl=nl, soc=soc)["E"]
    assert not st.any() and np.abs(E - ref).max() <= 1e-6
    assert max(np.abs(x.conj() @ x.T - np.eye(nb)).max() for x in X) <= 1e-8
