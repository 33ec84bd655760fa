"""The quaternion form of spin-orbit matrices of inversion-symmetric crystals (order N, each level once)
against the complex spinor matrix (order 2 N): the structure that it rests on, and the solves.

Bounds: FP64 energies 1e-10 eV and gradients 1e-8 of their scale (the parity bars), mixed energies
1e-6 eV. Eigenvector residuals 1e-9 eV: n eps |H| with n = 458, |H| ~ 170 eV is 2e-11, times a few for
inverse iteration. Orthonormality 1e-8, the projector bar."""
import ctypes as C

import numpy as np
import pytest

from ultimateepm_gb300 import _native as N
from ultimateepm_gb300 import api


def _ctx(orm, G, nl, prec, force_complex=False):
    m = api.Material("m", raw=N.UepmMaterial.from_buffer_copy(bytes(orm)))
    return api._Context(m, G, nl, True, prec, force_complex)


@pytest.mark.parametrize("key,quat", [("Si", True), ("Ge", True), ("GaAs", False)])
def test_the_spinor_matrix_is_quaternionic_without_antisymmetric_terms(oracle, mats, key, quat):
    """DD = conj(UU) and DU = -conj(UD), exactly, where the atoms are equal; not in a zinc-blende crystal."""
    G = oracle.generate_basis(8)
    n = len(G)
    ks = oracle.sample_first_bz(4, 3)
    for k in np.vstack([ks, [[0, 0, 0], [1, 0, 0], [0.5, 0.5, 0.5]]]) if quat else ks:
        for nl in (False, True):
            H = oracle.assemble(mats[key], G, k, nl=nl, soc=True)
            same = np.array_equal(H[n:, n:], H[:n, :n].conj()) and np.array_equal(H[n:, :n], -H[:n, n:].conj())
            assert same == quat


@pytest.mark.gpu
@pytest.mark.parametrize("key,shells,nl", [("Ge", 2, True), ("Ge", 3, True), ("Ge", 6, False), ("Si", 8, True),
                                           ("Ge", 9, True), ("Ge", 12, True), ("Ge", 13, True)])
@pytest.mark.parametrize("nb", [1, 7, 16])
def test_quaternion_solves_match_the_complex_ones(gpu, oracle, mats, key, shells, nl, nb):
    """Orders from 9 to 229 (65 and up leave ragged tiles; 181 and 229 start outside shared memory), even
    and odd band counts, values, vectors and gradients."""
    G = oracle.generate_basis(shells)
    nb = min(nb, 2 * len(G))
    ks = oracle.sample_first_bz(5, 11)
    E, g = {}, {}
    for fc in (True, False):
        ctx = _ctx(mats[key], G, nl, N.UEPM_PREC_FP64, fc)
        E[fc], X, g[fc], st = ctx.solve(ks, nb, vectors=True, gradient=True)
        assert not st.any()
        ctx.close()
    assert np.abs(E[True] - E[False]).max() <= 1e-10
    # one member of a pair has the pair's mean gradient, whichever vectors span it
    assert np.abs(g[True] - g[False]).max() <= 1e-8 * np.abs(g[True]).max()
    for q, k in enumerate(ks):
        H = oracle.assemble(mats[key], G, k, nl=nl, soc=True)
        V = X[q].T
        assert np.abs(H @ V - V * E[False][q]).max() <= 1e-9
        assert np.abs(V.conj().T @ V - np.eye(nb)).max() <= 1e-8
    if nb <= 16:
        ctx = _ctx(mats[key], G, nl, N.UEPM_PREC_MIXED)
        Em, _, gm, st = ctx.solve(ks, nb, gradient=True)
        assert not st.any() and np.abs(Em - E[True]).max() <= 1e-6
        ctx.close()


@pytest.mark.gpu
def test_one_plane_wave(gpu, oracle, mats):
    """The smallest quaternion matrix, 1 x 1: both levels are H_00."""
    G, ks = np.zeros((1, 3), dtype=np.int32), oracle.sample_first_bz(3, 5)
    for prec in (N.UEPM_PREC_FP64, N.UEPM_PREC_MIXED):
        ctx = _ctx(mats["Ge"], G, True, prec)
        E, _, _, st = ctx.solve(ks, 2)
        ctx.close()
        ref = [oracle.assemble(mats["Ge"], G, k, nl=True, soc=True)[0, 0].real for k in ks]
        assert not st.any() and np.abs(E - np.array(ref)[:, None]).max() <= 1e-10


@pytest.mark.gpu
def test_an_explicit_reduction_keeps_the_complex_matrix(gpu, oracle, mats):
    """uepm_tuning.reduction names a kernel of the complex matrix: the solve takes that one."""
    G, ks = oracle.generate_basis(8), oracle.sample_first_bz(4, 6)
    out = []
    for red in (0, 6):
        ctx = _ctx(mats["Ge"], G, True, N.UEPM_PREC_MIXED)
        N.check(gpu.uepm_ctx_set_tuning(ctx.h, C.byref(N.UepmTuning(reduction=red))))
        out.append(ctx.solve(ks, 12)[0])
        ctx.close()
    assert np.abs(out[0] - out[1]).max() <= 1e-6
