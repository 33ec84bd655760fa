"""What a solve answers when the CUDA runtime refuses a launch: a launcher that may give up leaves no error behind
and the other kernel runs; where there is no other kernel the solve fails, instead of going on from whatever the
workspace holds."""
import fake_runtime

GE = dict(material="Ge", shells=10, bands=8, nl=True, soc=True)


def test_the_fake_runtime_sees_an_ordinary_solve(native, tmp_path):
    (error, launches, _), = fake_runtime.run(tmp_path, dict(GE, k=10, mixed=True))
    assert error is None and any("k_tridiag_tri" in x[0] for x in launches) and any("k_bisect" in x[0] for x in launches)


def test_a_refused_quaternion_reduction_is_an_error(native, tmp_path):
    for refuse in ("occupancy k_tridiag_tri", "cudaFuncSetAttribute k_tridiag_tri", "launch k_tridiag_tri"):
        (error, launches, _), = fake_runtime.run(tmp_path, dict(GE, k=10, mixed=True, refuse=refuse))
        assert error is not None and not any("k_tridiag_tri" in x[0] for x in launches), refuse


def test_a_refused_launch_falls_back_without_an_error(native, tmp_path):
    tri = dict(material="GaAs", shells=12, bands=8, nl=True, k=10, mixed=True)  # complex order 181
    wide = dict(material="GaAs", shells=12, bands=8, nl=True, k=2)
    clus = dict(wide, tuning=dict(reduction=3))
    blocked = dict(material="GaAs", shells=10, bands=8, nl=True, soc=True, k=10, mixed=True)  # complex order 274
    tc = dict(material="GaAs", shells=10, bands=16, nl=True, soc=True, k=10, mixed=True)
    for case, refuse, other in ((tri, "cudaFuncSetAttribute k_tridiag_tri", "k_tridiag_fused"),
                                (tri, "occupancy k_tridiag_tri", "k_tridiag_fused"),
                                (wide, "launch k_tridiagINS_2cxIdEELi256ELi8ELb0ELi8E", "k_tridiagINS_2cxIdEELi256ELi8ELb0ELi1E"),
                                (clus, "cudaFuncSetAttribute k_tridiag_cluster", "k_tridiagINS_2cxIdEELi256ELi8ELb0ELi1E"),
                                (clus, "launch k_tridiag_cluster", "k_tridiagINS_2cxIdEELi256ELi8ELb0ELi1E"),
                                (blocked, "cudaFuncSetAttribute k_tridiag_blocked", "k_tridiag_fused"),
                                (tc, "cudaFuncSetAttribute k_refine_y_tc", "k_refine_project")):
        (_, plain, _), (error, launches, _) = fake_runtime.run(tmp_path, case, dict(case, refuse=refuse))
        name = refuse.split()[1]
        assert any(name in x[0] for x in plain) and not any(name in x[0] for x in launches), refuse
        assert any(other in x[0] for x in launches), refuse
        assert error is None, (refuse, error)
