"""The register-resident FP32 reduction of real and complex matrices at the edges of its 16-row blocks and of its
instantiations (1 to 12 blocks, complex 1 to 9): mixed energies against the oracle at the mixed bar of 1e-6 eV, on bases cut to
an arbitrary order, with the matrix read from memory (nonlocal) and formed from the local potential, and on free
electrons, whose columns are all without a reflector."""
import numpy as np
import pytest

from ultimateepm_gb300 import _native as N
from ultimateepm_gb300 import api

pytestmark = pytest.mark.gpu


def _check(oracle, mat, n, nl, real=True):
    G = np.ascontiguousarray(oracle.generate_basis(13)[:n])
    ks = oracle.sample_first_bz(3, 5)
    nb = min(n, 6)
    ctx = api._Context(api.Material("m", raw=N.UepmMaterial.from_buffer_copy(bytes(mat))), G, nl, False, N.UEPM_PREC_MIXED)
    assert ctx.real == real
    E, _, _, st = ctx.solve(np.tile(ks, (210, 1)), nb)
    ctx.close()
    assert not st.any()
    assert np.abs(E[:3] - oracle.band_structure(mat, G, ks, nb, nl=nl, soc=False)["E"]).max() <= 1e-6
    assert np.array_equal(E, np.tile(E[:3], (210, 1)))


@pytest.mark.parametrize("nl", [False, True])
@pytest.mark.parametrize("n", [1, 2, 15, 16, 17, 33, 48, 64, 65, 80, 81, 96, 97, 113, 128, 129, 144, 145, 160, 176, 177, 192])
def test_orders_at_the_block_edges(gpu, oracle, mats, n, nl):
    _check(oracle, mats["Si"], n, nl)


@pytest.mark.parametrize("n", [16, 63, 137])
def test_columns_without_a_reflector(gpu, oracle, mats, n):
    m = type(mats["Si"]).from_buffer_copy(bytes(mats["Si"]))
    m.V3S = m.V4S = m.V8S = m.V11S = 0.0
    _check(oracle, m, n, False)


@pytest.mark.parametrize("nl", [False, True])
@pytest.mark.parametrize("n", [1, 2, 15, 16, 17, 33, 49, 65, 81, 96, 97, 112, 113, 128, 129, 144, 145])
def test_complex_orders_at_the_block_edges(gpu, oracle, mats, n, nl):
    _check(oracle, mats["InP"], n, nl, real=False)
