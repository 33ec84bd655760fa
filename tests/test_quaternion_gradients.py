"""Gradients of mixed spin-orbit solves in quaternion form against the FP64 solve of the complex matrix, for Kramers
pairs more than 1e-3 eV from their neighbours. Bound: the FP32 vectors miss the subspace by a few eps32 |H| / gap, with |H|
about 170 eV and 1 eV to the states beyond the guard bands 3e-5, which enters the gradient to first order:
1e-4 of the largest gradient."""
import numpy as np
import pytest

from ultimateepm_gb300 import _native as N
from ultimateepm_gb300 import api

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("key,shells,nl", [("Ge", 3, True), ("Ge", 6, False), ("Si", 8, True), ("Ge", 9, True), ("Ge", 12, True), ("Ge", 13, True)])
@pytest.mark.parametrize("nb", [1, 7, 16])
def test_mixed_gradients(gpu, oracle, mats, key, shells, nl, nb):
    G, ks = oracle.generate_basis(shells), oracle.sample_first_bz(5, 11)
    nb = min(nb, 2 * len(G))
    out = []
    for prec, fc, want in ((N.UEPM_PREC_FP64, True, min(nb + 2, 2 * len(G))), (N.UEPM_PREC_MIXED, False, nb)):
        ctx = api._Context(api.Material(key, raw=N.UepmMaterial.from_buffer_copy(bytes(mats[key]))), G, nl, True, prec, fc)
        E, _, g, st = ctx.solve(ks, want, gradient=True)
        ctx.close()
        assert not st.any()
        out.append((E, g))
    (E, g), (Em, gm) = out
    assert np.abs(Em - E[:, :nb]).max() <= 1e-6
    seen = 0
    for q in range(len(ks)):
        for b in range(nb):
            p = b // 2 * 2  # the pair's first band
            if (p > 0 and E[q, p] - E[q, p - 1] < 1e-3) or (p + 2 < E.shape[1] and E[q, p + 2] - E[q, p] < 1e-3):
                continue
            seen += 1
            assert np.abs(gm[q, b] - g[q, b]).max() <= 1e-4 * np.abs(g).max()
    assert seen > 0
