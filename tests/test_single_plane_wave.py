"""A basis of one plane wave: the mixed solver's padded products of one matrix must not reach its neighbour's."""
import numpy as np
import pytest

from ultimateepm_gb300 import _native as N
from ultimateepm_gb300 import api

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("key,nl", [("Si", False), ("Si", True), ("InP", True)])
def test_one_plane_wave_per_matrix(gpu, oracle, mats, key, nl):
    G = np.ascontiguousarray(oracle.generate_basis(5)[:1])
    ks = oracle.sample_first_bz(3, 5)
    ctx = api._Context(api.Material("m", raw=N.UepmMaterial.from_buffer_copy(bytes(mats[key]))), G, nl, False, N.UEPM_PREC_MIXED)
    E, _, _, st = ctx.solve(np.tile(ks, (1000, 1)), 1)
    ctx.close()
    assert not st.any()
    assert np.abs(E - np.tile(oracle.band_structure(mats[key], G, ks, 1, nl=nl, soc=False)["E"], (1000, 1))).max() <= 1e-6
