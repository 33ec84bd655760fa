"""Every kernel gets the shared memory that its launch asks for, at every order: the 48 KB that a kernel has without
asking hold its static shared memory too."""
import numpy as np
import pytest

import fake_runtime
from ultimateepm_gb300 import _native as N
from ultimateepm_gb300 import api

# FP64 vectors of 10 or 11 words per row cross 48 KB at quaternion orders 140 and 153, complex 279 and 307
ORDERS = [*range(136, 157), *range(272, 312, 1)]


@pytest.mark.parametrize("mixed", [False, True])
def test_every_order_is_launched(native, tmp_path, mixed):
    cases = [dict(material="GaAs" if form == "complex" else "Ge", shells=22, plane_waves=n, bands=4, k=k, nl=False, soc=form == "quaternion", mixed=mixed,
                  vectors=True) for n in ORDERS for form in ("real", "complex", "quaternion") for k in (2, 100) if n < 257 or form != "quaternion"]
    got = fake_runtime.run(tmp_path, *cases)
    assert [(c["plane_waves"], c["material"], c["soc"], c["k"], e) for c, (e, _, _) in zip(cases, got) if e] == []


@pytest.mark.gpu
@pytest.mark.parametrize("key,soc,n", [("Ge", True, 153), ("GaAs", False, 306), ("GaAs", False, 307)])
def test_fp64_solves_at_the_line(gpu, oracle, mats, key, soc, n):
    """One CTA per matrix (78 of them): energies within the FP64 bar of 1e-10 eV of the oracle."""
    G, ks = oracle.generate_basis(22)[:n], oracle.sample_first_bz(2, 9)
    ctx = api._Context(api.Material(key, raw=N.UepmMaterial.from_buffer_copy(bytes(mats[key]))), G, False, soc)
    E, _, _, st = ctx.solve(np.tile(ks, (39, 1)), 8)
    ctx.close()
    ref = oracle.band_structure(mats[key], G, ks, 8, nl=False, soc=soc)["E"]
    assert not st.any() and np.abs(E - np.tile(ref, (39, 1))).max() <= 1e-10


def test_a_kernel_has_one_limit(native, tmp_path):
    """The limit is the process's: at every order the same, so that a thread that solves a small order between another
    thread's limit and its launch does not take shared memory from it."""
    every = [dict(material=key, shells=s, bands=nb, k=k, nl=nl, soc=soc, mixed=mixed, vectors=True, tuning=dict(reduction=red))
             for key, nl, soc in (("Ge", True, True), ("GaAs", True, True), ("InP", True, False), ("Ge", True, False)) for s in (6, 10, 13)
             for nb, k in ((4, 2), (28, 100)) for mixed in (False, True) for red in ((0, 3, 6) if mixed else (0, 2))]
    limits = {}
    for _, launches, smem in fake_runtime.run(tmp_path, *every):
        for kernel, most in smem:
            limits.setdefault(kernel, set()).add(most)
    assert len(limits) > 10 and {k: v for k, v in limits.items() if len(v) > 1} == {}
