"""uepm_tuning on spin-orbit contexts that are solved in quaternion form (order N, half the matrix's): vector_lanes chooses
the back-transformation's kernel where the rows fit, as for the other forms, with the same results."""
import ctypes as C

import numpy as np
import pytest

import fake_runtime
from ultimateepm_gb300 import _native as N
from ultimateepm_gb300 import api


@pytest.mark.parametrize("mixed", [False, True])
def test_vector_lanes_are_honoured(native, tmp_path, mixed):
    # (shells, lanes asked for): lanes taken; orders 89, 137, 181 and 229, at most 12 rows per lane
    want = {(8, 0): 8, (8, 8): 8, (8, 16): 16, (8, 32): 32, (10, 0): 16, (10, 8): 16, (10, 32): 32, (12, 16): 16, (12, 32): 32, (13, 0): 32, (13, 16): 32}
    cases = [dict(material="Ge", shells=s, bands=4, k=3, nl=True, soc=True, mixed=mixed, vectors=True, tuning=dict(vector_lanes=v)) for s, v in want]
    for (key, lanes), (error, launches, _) in zip(want.items(), fake_runtime.run(tmp_path, *cases)):
        got = [x[0] for x in launches if "k_backtransform" in x[0]]
        assert error is None and len(got) == 1 and f"2qtI{'f' if mixed else 'd'}EELi{lanes}E" in got[0], (key, got)


@pytest.mark.gpu
@pytest.mark.parametrize("shells", [8, 10, 12])
def test_every_lane_count_gives_the_same_levels(gpu, oracle, mats, shells):
    G, ks = oracle.generate_basis(shells), oracle.sample_first_bz(3, 5)
    ref = oracle.band_structure(mats["Ge"], G, ks, 9, nl=True, soc=True)["E"]
    for prec, tol in ((N.UEPM_PREC_FP64, 1e-10), (N.UEPM_PREC_MIXED, 1e-6)):
        for lanes in (0, 8, 16, 32):
            ctx = api._Context(api.Material("Ge", raw=N.UepmMaterial.from_buffer_copy(bytes(mats["Ge"]))), G, True, True, prec)
            N.check(gpu.uepm_ctx_set_tuning(ctx.h, C.byref(N.UepmTuning(vector_lanes=lanes))))
            E, X, _, st = ctx.solve(ks, 9, vectors=True)
            ctx.close()
            assert not st.any() and np.abs(E - ref).max() <= tol
            assert max(np.abs(x.conj() @ x.T - np.eye(9)).max() for x in X) <= 1e-8
