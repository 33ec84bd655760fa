"""The scalars of the Householder reductions (sqrt_pair and recip, uepm_common.cuh; reflector, tridiag_reg.cu), refined from
hardware approximations, through uepm_reflector_scalars_device.

FP64 bounds, u = 2^-53: the approximations are within 2^-19.9, so that the third-order steps leave (5 / 16) 2^-56.7 =
2^-58.4 of the root's reciprocal and 2^-59.7 of the reciprocal. The root ends with a correction by its residual: u. The
reciprocal: u and the step's 2^-59.7: 1.02 u. The root's reciprocal takes half the rounding of x y besides: 1.53 u.
Outside the exponents that the approximations take (in_seed_range), CUDA's root and quotient, exactly.

FP32 bounds, v = 2^-24: |alpha|^2 + |tail|^2 is rounded once (real) or up to three times (complex), so that beta is
within 1.5 v or 2.5 v (half of that, and its own rounding), tau's real part d / |beta|, d = |Re alpha| + |beta|, within
half of beta's error and two roundings, 2.75 v and 3.25 v, its imaginary part within beta's error and one
rounding, 3.5 v; 1 / (alpha - beta) within d's error and two roundings, 4.5 v real, and complex within
three times d's error of 3.5 v and four roundings, 14.5 v of its magnitude. Each 1 % more for terms of second order. The
errors of beta and tau (real) have no common sign: means below v / 20 (with rounded approximations alone, whose bias moved
refined eigenvalues, they are not)."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
U, V = 2.0 ** -53, 2.0 ** -24


def _run(gpu, fn, *x):
    import torch

    n = len(x[0])
    dx = torch.from_numpy(np.ascontiguousarray(np.stack([x[0], x[1] if len(x) > 2 else np.zeros(n), x[-1]]))).cuda()
    dy = torch.full((5, n), float("nan"), dtype=torch.float64, device="cuda")
    assert gpu.uepm_reflector_scalars_device(fn, C.c_void_p(dx.data_ptr()), n, C.c_void_p(dy.data_ptr()), None) == 0
    torch.cuda.synchronize()
    return dy.cpu().numpy()


def test_fp64_root_and_reciprocals_over_the_range(gpu):
    rng = np.random.default_rng(2)
    x = np.concatenate([np.ldexp(rng.uniform(0.5, 1.0, 400000), rng.integers(-821, 776, 400000)), np.linspace(1.0, 4.0, 100001)])
    y = _run(gpu, 0, x, x)
    w = np.asarray(x, dtype=np.longdouble)
    root = np.sqrt(w)
    for got, want, bound in ((y[0], root, 1.0), (y[1], 1 / root, 1.53), (y[2], 1 / w, 1.02)):
        assert float(np.abs(got / want - 1).max()) <= 1.01 * bound * U
    assert np.array_equal(_run(gpu, 0, -x, -x)[2], -y[2])


def test_fp64_outside_the_range_is_cudas_root_and_quotient(gpu):
    import torch

    rng = np.random.default_rng(3)
    x = np.concatenate([np.ldexp(rng.uniform(0.5, 1.0, 2000), rng.integers(-1021, -823, 2000)), np.ldexp(rng.uniform(0.5, 1.0, 2000), rng.integers(779, 1024, 2000)),
                        [5e-324, 1e-310, 2.0 ** -1022, 2.0 ** -823, 2.0 ** 777, 1.7e308, np.inf, np.nan, 0.0]])
    y = _run(gpu, 0, x, x)
    t = torch.from_numpy(x).cuda()
    root = torch.sqrt(t)
    for got, want in ((y[0], root), (y[1], 1.0 / root), (y[2], 1.0 / t)):
        assert np.array_equal(got, want.cpu().numpy(), equal_nan=True)


def _columns(n, spread):
    rng = np.random.default_rng(4)
    e = rng.integers(-spread, spread + 1, (3, n))
    f = np.ldexp(rng.uniform(0.5, 1.0, (3, n)), e) * np.where(rng.random((3, n)) < 0.5, -1, 1)
    near = np.ldexp(rng.uniform(0.5, 1.0, (2, n)), e[:1] + rng.integers(-2, 3, (2, n)))  # comparable parts
    f[1:, ::2] = near[:, ::2]
    return (f[0].astype(np.float32).astype(float), f[1].astype(np.float32).astype(float), (f[2] ** 2).astype(np.float32).astype(float))


def test_fp32_real_reflectors(gpu):
    al, _, ss = _columns(1000000, 25)
    y = _run(gpu, 1, al, ss)
    s = np.sqrt(al * al + ss)
    beta = np.where(al >= 0, -s, s)
    errs = [(y[0] / beta - 1) / V, (y[1] / ((beta - al) / beta) - 1) / V, (y[3] * (al - beta) - 1) / V]
    for e, bound in zip(errs, (1.5, 2.75, 4.5)):
        assert np.abs(e).max() <= 1.01 * bound
    assert abs(errs[0].mean()) <= 0.05 and abs(errs[1].mean()) <= 0.05


def test_fp32_complex_reflectors(gpu):
    ar, ai, ss = _columns(1000000, 25)
    y = _run(gpu, 2, ar, ai, ss)
    s = np.sqrt(ar * ar + ai * ai + ss)
    beta = np.where(ar >= 0, -s, s)
    tau = (beta - (ar + 1j * ai)) / beta
    assert (np.abs(y[0] / beta - 1).max() <= 2.525 * V) and (np.abs(y[1] / tau.real - 1).max() <= 1.01 * 3.25 * V)
    assert np.abs(y[2] / tau.imag - 1).max() <= 1.01 * 3.5 * V
    sc = 1 / (ar + 1j * ai - beta)
    assert (np.abs(y[3] + 1j * y[4] - sc) / np.abs(sc)).max() <= 1.01 * 14.5 * V


def test_fp32_columns_without_a_tail_and_non_finite_ones(gpu):
    tiny = float(np.finfo(np.float32).tiny)
    al, ss = np.array([3.0, -2.0, 0.0, 1e-30, 5.0]), np.array([0.0, 0.0, 0.0, tiny, tiny / 2])
    y = _run(gpu, 1, al, ss)
    assert np.array_equal(y[0], al.astype(np.float32)) and not y[1].any() and not y[3].any()
    assert np.array_equal(_run(gpu, 2, al, np.zeros(5), ss)[:, :], y)
    bad = np.array([np.inf, 1.0, np.nan, 1e30])
    y = _run(gpu, 1, bad, np.array([1.0, np.inf, 1.0, 1.0]))
    assert not np.isfinite(y[0]).any()  # the matrix's status
