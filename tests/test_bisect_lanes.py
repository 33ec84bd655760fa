"""The bisection gives a value 1 to 32 lanes by how many values the batch holds (launch_bisect). Each choice
visits the brackets of the one-lane bisection, so a k-point's energies are the same bits in every batch
size: compared here across all the choices, and with the oracle at the FP64 bar of 1e-10 eV."""
import numpy as np
import pytest

from ultimateepm_gb300 import _native as N
from ultimateepm_gb300 import api

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [N.UEPM_PREC_FP64, N.UEPM_PREC_MIXED])
@pytest.mark.parametrize("shells,nb", [(4, 15), (5, 7), (6, 16)])
def test_every_batch_size_gives_the_same_bits(gpu, oracle, mats, prec, shells, nb):
    G = oracle.generate_basis(shells)
    nb = min(nb, len(G))
    ks = oracle.sample_first_bz(2, 9)
    ctx = api._Context(api.Material("Si", raw=N.UepmMaterial.from_buffer_copy(bytes(mats["Si-CB"]))), G, False, False, prec)
    first = np.concatenate([ctx.solve(k, nb)[0] for k in ks])  # 32 lanes
    tol = 1e-10 if prec == N.UEPM_PREC_FP64 else 1e-6
    assert np.abs(first - oracle.band_structure(mats["Si-CB"], G, ks, nb)["E"]).max() <= tol
    # values per batch on both sides of every threshold of either precision
    for values in (500, 700, 2000, 5000, 9000, 20000, 39000, 41000):
        nk = values // nb
        E, _, _, st = ctx.solve(np.tile(ks, (nk // 2 + 1, 1)), nb)
        assert not st.any()
        assert np.array_equal(E[:2], first) and np.array_equal(E[-2:], first)
        assert np.array_equal(E, np.tile(first, (nk // 2 + 1, 1)))
    ctx.close()


def test_all_values_of_one_matrix(gpu, oracle, mats):
    """Every value of one matrix, in CTAs of a few values each."""
    G = oracle.generate_basis(8)
    ks = oracle.sample_first_bz(1, 4)
    ctx = api._Context(api.Material("Si", raw=N.UepmMaterial.from_buffer_copy(bytes(mats["Si-CB"]))), G, False, False)
    E = ctx.solve(ks, len(G))[0]
    ctx.close()
    assert np.abs(E - oracle.band_structure(mats["Si-CB"], G, ks, len(G))["E"]).max() <= 1e-10
