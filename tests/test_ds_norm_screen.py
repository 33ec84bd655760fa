"""The FP32 screen of the double-single assembly's FP64 tests: k-points beside high-symmetry ones, where pairs of
norms |k + G| differ by relative amounts on both sides of its bounds (2e-5) and of the FP64 element's (1e-5), square
and gaussian wells, with and without spin-orbit coupling: mixed energies against the FP64 path, which forms every element
in FP64, at the mixed bar of 1e-6 eV. (Not against the CPU oracle: at the smallest differences the reference's formula
divides two rounding errors, and its own FP64 evaluations differ by more than that.)"""
import numpy as np
import pytest

from ultimateepm_gb300 import _native as N
from ultimateepm_gb300 import api

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("key,soc", [("Si", False), ("Ge", False), ("InP", False), ("GaAs", True), ("Ge", True)])
def test_norm_differences_at_the_bounds(gpu, oracle, mats, key, soc):
    G = oracle.generate_basis(7)
    eps = [0.0, 1e-9, 3e-7, 3e-6, 0.9e-5, 1.1e-5, 1.9e-5, 2.1e-5, 4e-5, 1e-4, 1e-3]
    ks = np.array([np.array(k0) + np.array([e, 0.0, 0.0]) for k0 in ((0, 0, 0), (0.5, 0.5, 0.0), (0.25, 0.25, 0.25)) for e in eps])
    E = []
    for prec in (N.UEPM_PREC_MIXED, N.UEPM_PREC_FP64):
        ctx = api._Context(api.Material(key, raw=N.UepmMaterial.from_buffer_copy(bytes(mats[key]))), G, True, soc, prec)
        e, _, _, st = ctx.solve(ks, 10)
        ctx.close()
        assert not st.any()
        E.append(e)
    assert np.abs(E[0] - E[1]).max() <= 1e-6
