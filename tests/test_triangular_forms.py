"""Which form of the triangular reduction (tridiag_tri.cu) each order takes: CTAs of 128, 256 or 512 threads and, where the
triangle does not fit an SM, its first columns in global memory. Every form that the library holds is reached."""
import re

import fake_runtime


def test_every_form_is_reached_and_by_its_orders(native, tmp_path):
    cases = [dict(material="Ge", shells=22, plane_waves=n, bands=2, k=2, soc=True, mixed=True) for n in (1, 2, 74, 75, 109, 110, 159, 160, 256)]
    cases += [dict(material="InP", shells=22, plane_waves=n, bands=2, k=2, mixed=True) for n in (174, 175, 215, 230, 231)]
    seen = []
    for c, (error, launches, _) in zip(cases, fake_runtime.run(tmp_path, *cases)):
        form = [re.search(r"k_tridiag_triINS_2(\w)tIfEELi(\d+)ELi\dELb(\d)E|k_tridiag_triINS_2(c)xIfEELi(\d+)ELi\dELb(\d)E", x[0]) for x in launches]
        form = [tuple(g for g in m.groups() if g) for m in form if m]
        assert error is None and len(form) <= 1
        seen.append((c["plane_waves"], *form))
    q = [(n, ("q", t, s)) for n, t, s in ((1, "128", "0"), (2, "128", "0"), (74, "128", "0"), (75, "256", "0"), (109, "256", "0"), (110, "512", "0"),
                                          (159, "512", "0"), (160, "512", "1"), (256, "512", "1"))]
    assert seen == q + [(174,), (175, ("c", "512", "0")), (215, ("c", "512", "0")), (230, ("c", "512", "1")), (231,)]
    assert sum("k_tridiag_tri" in k for k in fake_runtime.kernels(tmp_path)) == len({f for _, *fs in seen for f in fs})
