"""Which form the bisection takes (launch_bisect): lanes per value by the number of values, and, where the CTA's
matrices do not fit its shared memory, the next form with more lanes, not at once the one with 32. Every form
gives the same bits."""
import numpy as np
import pytest

import fake_runtime
from ultimateepm_gb300 import _native as N
from ultimateepm_gb300 import api

# (shells, nl, soc, mixed, bands, k) of Ge: the lanes per value, and those of the FP64 phase
FORMS = [((10, False, False, False, 16, 3000), (1, 1)),     # n = 137, 48000 values, 9 matrices per CTA
         ((10, False, False, False, 4, 11000), (4, 1)),     # 33 matrices (145 KB) do not fit: 9 do
         ((10, False, False, False, 2, 21000), (4, 1)),
         ((10, False, False, False, 1, 14000), (8, 8)),     # 32 matrices of 4 lanes do not fit either
         ((10, False, False, False, 1, 3000), (8, 8)),
         ((10, False, False, False, 1, 30), (32, 32)),
         ((12, False, False, False, 4, 11000), (4, 1)),     # 181
         ((13, True, True, False, 16, 2500), (4, 1)),       # quaternion 229: 8 values per matrix
         ((13, True, True, False, 1, 2500), (16, 16)),
         ((12, False, False, True, 1, 8000), (1, 1)),       # FP32, 5 vectors per matrix
         ((12, False, False, True, 1, 900), (8, 8))]


def test_the_next_form_stands_in_where_one_does_not_fit(native, tmp_path):
    cases = [dict(material="Ge", shells=s, nl=nl, soc=soc, mixed=mixed, bands=nb, k=k, tuning=dict(streams=1)) for (s, nl, soc, mixed, nb, k), _ in FORMS]
    for (case, (p, q)), (error, launches, _) in zip(FORMS, fake_runtime.run(tmp_path, *cases)):
        got = [x for x in launches if "k_bisect" in x[0]]
        assert error is None and len(got) == 1
        assert f"k_bisectI{'f' if case[3] else 'd'}Li{p}ELi{q}E" in got[0][0], (case, got)


@pytest.mark.gpu
@pytest.mark.parametrize("shells,nb,nk", [(10, 1, 14000), (10, 2, 20500), (10, 4, 10250), (12, 3, 14000)])
def test_many_values_of_few_bands_are_the_same_bits(gpu, oracle, mats, shells, nb, nk):
    """More than 40000 FP64 values (and 14000 of one band), orders 137 and 181, against single k-points."""
    G, ks = oracle.generate_basis(shells), oracle.sample_first_bz(2, 9)
    ctx = api._Context(api.Material("Si", raw=N.UepmMaterial.from_buffer_copy(bytes(mats["Si-CB"]))), G, False, False)
    first = np.concatenate([ctx.solve(k, nb)[0] for k in ks])
    E, _, _, st = ctx.solve(np.tile(ks, (nk // 2, 1)), nb)
    ctx.close()
    assert not st.any() and np.array_equal(E, np.tile(first, (nk // 2, 1)))
    assert np.abs(first - oracle.band_structure(mats["Si-CB"], G, ks, nb)["E"]).max() <= 1e-10
