"""The Rayleigh-Ritz product on the tensor cores against the FP32 pipe, at orders and band counts on both sides of the
line that the automatic choice draws (orders 89 to 229, 5 to 28 bands; 113 at 16 bands, 89 at 28 and 181 at 16 lie on
the tensor cores' side): energies within 1e-9 eV of each other and within the mixed bar of 1e-6 eV of the oracle."""
import ctypes as C

import numpy as np
import pytest

from ultimateepm_gb300 import _native as N
from ultimateepm_gb300 import api

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("key,shells,nb", [("InP", 8, 12), ("InP", 8, 28), ("InP", 9, 12), ("InP", 9, 16), ("InP", 10, 16),
                                           ("InP", 10, 28), ("InP", 12, 5), ("InP", 12, 16), ("InAs", 13, 8), ("InAs", 13, 12)])
def test_both_forms_agree_across_the_line(gpu, oracle, mats, key, shells, nb):
    G = oracle.generate_basis(shells)
    ks = oracle.sample_first_bz(7, 44)
    out = []
    for tc in (0, 1):
        ctx = api._Context(api.Material(key, raw=N.UepmMaterial.from_buffer_copy(bytes(mats[key]))), G, True, False,
                           N.UEPM_PREC_MIXED)
        N.check(gpu.uepm_ctx_set_tuning(ctx.h, C.byref(N.UepmTuning(tensor_cores=tc))))
        E, _, _, st = ctx.solve(ks, nb)
        ctx.close()
        assert not st.any()
        out.append(E)
    ref = oracle.band_structure(mats[key], G, ks, nb, nl=True, soc=False)["E"]
    assert np.abs(out[0] - out[1]).max() <= 1e-9
    assert np.abs(out[0] - ref).max() <= 1e-6
