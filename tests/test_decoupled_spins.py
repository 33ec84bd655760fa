"""Spin-orbit contexts without spin-orbit strength (mu_soc = 0): H = diag(h, h), solved on the scalar matrix h.
The structure on the CPU, and the solves against the full complex matrix (force_complex): FP64 energies within
1e-10 eV, gradients within 1e-8 of their scale, mixed energies within 1e-6 eV; vectors as eigenvectors of the full
matrix (residual 1e-9 eV, orthonormality 1e-8)."""
import numpy as np
import pytest

from ultimateepm_gb300 import _native as N
from ultimateepm_gb300 import api


def _ctx(orm, G, nl, prec, force_complex=False):
    m = api.Material("m", raw=N.UepmMaterial.from_buffer_copy(bytes(orm)))
    return api._Context(m, G, nl, True, prec, force_complex)


@pytest.mark.parametrize("key,zero", [("Si", True), ("GaP", True), ("Ge", False), ("GaAs", False)])
def test_the_spins_decouple_exactly_without_spin_orbit_strength(oracle, mats, key, zero):
    assert (mats[key].mu_soc == 0.0) == zero
    G = oracle.generate_basis(8)
    n = len(G)
    for k in oracle.sample_first_bz(3, 5):
        for nl in (False, True):
            H = oracle.assemble(mats[key], G, k, nl=nl, soc=True)
            h = oracle.assemble(mats[key], G, k, nl=nl, soc=False)
            same = not H[:n, n:].any() and np.array_equal(H[:n, :n], h) and np.array_equal(H[n:, n:], h)
            assert same == zero


@pytest.mark.gpu
@pytest.mark.parametrize("key,shells,nl", [("Si", 6, False), ("Si", 8, True), ("GaP", 8, True), ("GaP", 10, False)])
@pytest.mark.parametrize("nb", [1, 9, 16])
def test_scalar_solves_match_the_full_matrix(gpu, oracle, mats, key, shells, nl, nb):
    G = oracle.generate_basis(shells)
    ks = oracle.sample_first_bz(5, 12)
    E, g = {}, {}
    for fc in (True, False):
        ctx = _ctx(mats[key], G, nl, N.UEPM_PREC_FP64, fc)
        E[fc], X, g[fc], st = ctx.solve(ks, nb, vectors=True, gradient=True)
        assert not st.any()
        ctx.close()
    assert np.abs(E[True] - E[False]).max() <= 1e-10
    assert np.abs(g[True] - g[False]).max() <= 1e-8 * np.abs(g[True]).max()
    for q, k in enumerate(ks):
        H, V = oracle.assemble(mats[key], G, k, nl=nl, soc=True), X[q].T
        assert np.abs(H @ V - V * E[False][q]).max() <= 1e-9
        assert np.abs(V.conj().T @ V - np.eye(nb)).max() <= 1e-8
    ctx = _ctx(mats[key], G, nl, N.UEPM_PREC_MIXED)
    Em, Xm, _, st = ctx.solve(np.tile(ks, (300, 1)), nb, vectors=True)  # two lanes
    ctx.close()
    assert not st.any() and np.abs(Em[:5] - E[True]).max() <= 1e-6
    assert np.array_equal(Em, np.tile(Em[:5], (300, 1)))
    V = Xm[-1].T
    assert np.abs(V.conj().T @ V - np.eye(nb)).max() <= 1e-8


@pytest.mark.gpu
def test_every_level_of_a_decoupled_matrix(gpu, oracle, mats):
    """nb = 2 N, through the host API, energies doubled in order."""
    G, ks = oracle.generate_basis(4), oracle.sample_first_bz(2, 3)
    ctx = _ctx(mats["GaP"], G, True, N.UEPM_PREC_FP64)
    E = ctx.solve(ks, 2 * len(G))[0]
    ctx.close()
    ref = oracle.band_structure(mats["GaP"], G, ks, 2 * len(G), nl=True, soc=True)["E"]
    assert np.array_equal(E[:, ::2], E[:, 1::2]) and np.abs(E - ref).max() <= 1e-10
