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


def test_the_autotuner_times_what_changes_the_solve(native, tmp_path):
    """Shapes timed (three solves each; every shape takes the same time here, so the first stands): the automatic one, the
    reductions, and of the other fields those that the automatic reduction takes."""
    ge, inp, si = dict(material="Ge", nl=True, soc=True), dict(material="InP", nl=True), dict(material="Si")
    want = [(dict(ge, shells=8, mixed=True), 1 + 5 + 3),      # quaternion 89 in shared memory: lanes of 8, 16, 32
            (dict(ge, shells=10, mixed=True), 1 + 5 + 2),     # 137: lanes of 16, 32
            (dict(ge, shells=8), 1 + 2 + 5),                  # FP64, global memory: CTAs per SM; no vectors, no lanes
            (dict(inp, shells=9, mixed=True), 1 + 5 + 3),     # complex 113 in registers
            (dict(inp, shells=12, mixed=True), 1 + 5 + 3),    # complex 181, triangular
            (dict(inp, shells=11, mixed=True), 1 + 5 + 5 + 3),  # complex 169, deferred
            (dict(si, shells=12, mixed=True), 1 + 5 + 3),     # real 181 in registers
            (dict(si, shells=13, mixed=True), 1 + 5 + 5 + 3)]  # real 229, deferred
    for (case, shapes), (error, launches, _) in zip(want, fake_runtime.run(tmp_path, *[dict(c, bands=4, k=1, autotune=200) for c, _ in want])):
        solves = sum("k_rows" in x[0] for x in launches) - 1  # the solve itself
        assert error is None and solves == 3 * shapes, (case, solves)
