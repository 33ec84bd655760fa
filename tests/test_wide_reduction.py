"""The FP64 reduction with a cluster of 8, 4 or 2 CTAs per matrix (batches of at most half as many matrices as
SMs): energies and gradients are the same bits as with one CTA per matrix, whatever the batch, and within the
FP64 bar of 1e-10 eV of the oracle. Orders: real, complex and quaternion; 65, 89 and 113 with ragged last
chunks (1, 25 and 17 rows), 181, and 274 beyond the smaller instantiation."""
import numpy as np
import pytest

from ultimateepm_gb300 import _native as N
from ultimateepm_gb300 import api

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("key,shells,nl,soc", [("Si-CB", 9, False, False), ("Si-CB", 12, False, False), ("GaAs", 8, True, False),
                                               ("GaAs", 10, True, True), ("Ge", 7, True, True), ("Ge", 12, True, True)])
def test_cluster_sizes_give_the_same_bits(gpu, oracle, mats, key, shells, nl, soc):
    G = oracle.generate_basis(shells)
    ks = oracle.sample_first_bz(2, 31)
    ctx = api._Context(api.Material(key, raw=N.UepmMaterial.from_buffer_copy(bytes(mats[key]))), G, nl, soc)
    out = [ctx.solve(np.tile(ks, (nk // 2, 1)), 9, gradient=True) for nk in (2, 16, 18, 32, 34, 64, 100, 170)]
    ctx.close()
    ref = oracle.band_structure(mats[key], G, ks, 9, nl=nl, soc=soc)["E"]
    assert np.abs(out[0][0] - ref).max() <= 1e-10
    for E, _, g, st in out:
        assert not st.any()
        assert np.array_equal(E, np.tile(out[0][0], (len(E) // 2, 1)))
        assert np.array_equal(g, np.tile(out[0][2], (len(E) // 2, 1, 1)))
