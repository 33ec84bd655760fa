"""The Rayleigh-Ritz product on the tensor cores against the FP32 pipe where both are known to run: the kernel counts
of the two solves differ by the product's own launch. Complex matrices under one reduction (5), and quaternionic ones as
the automatic choice solves them (only the first half of H and Y formed, one or two row tiles, ragged at orders 113,
137, 181 and 229): energies within 1e-9 eV of each other and within the mixed bar of 1e-6 eV of the oracle."""
import ctypes as C

import numpy as np
import pytest

from ultimateepm_gb300 import _native as N
from ultimateepm_gb300 import api

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("key,shells,nl,soc,nb,red", [("GaP", 8, False, True, 16, 5), ("GaAs", 8, True, True, 16, 5), ("InP", 12, True, False, 14, 5),
                                                      ("Ge", 9, True, True, 16, 0), ("Ge", 10, True, True, 16, 0), ("Ge", 12, True, True, 13, 0),
                                                      ("Ge", 12, True, True, 16, 0), ("Ge", 13, False, True, 24, 0)])
def test_the_product_on_either_pipe(gpu, oracle, mats, key, shells, nl, soc, nb, red):
    G, ks = oracle.generate_basis(shells), oracle.sample_first_bz(7, 43)
    E, launches = [], []
    for tc in (0, 1):
        ctx = api._Context(api.Material(key, raw=N.UepmMaterial.from_buffer_copy(bytes(mats[key]))), G, nl, soc, N.UEPM_PREC_MIXED)
        N.check(gpu.uepm_ctx_set_tuning(ctx.h, C.byref(N.UepmTuning(reduction=red, tensor_cores=tc))))
        before = gpu.uepm_kernel_launches()
        e, _, _, st = ctx.solve(ks, nb)
        launches.append(gpu.uepm_kernel_launches() - before)
        ctx.close()
        assert not st.any()
        E.append(e)
    assert launches[0] == launches[1] + 1
    assert np.abs(E[0] - E[1]).max() <= 1e-9
    assert np.abs(E[0] - oracle.band_structure(mats[key], G, ks, nb, nl=nl, soc=soc)["E"]).max() <= 1e-6
