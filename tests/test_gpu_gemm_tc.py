"""The FP64 GEMM on the tensor cores (exact integer digit products), through qk_dgemm_dev with the
context setting dgemm_path = 3.

The result is the exact product of the operands' 62-bit row-scaled integers, rounded once per k
slice (at most 16 slices are added in FP64), so
  |C - AB| <= 17 * 2^-53 sum_k |a_ik b_kj| + k * 2^-59 max_k |a_ik| max_k |b_kj|
whatever the sizes; small integers come out exactly.
"""
from fractions import Fraction

import numpy as np
import pytest

from quack_gb300 import api

pytestmark = pytest.mark.gpu


@pytest.fixture()
def tc():
    c = api.Context(0)
    for b in range(40):
        c.tune_set("dgemm_path", 2 ** b, 3)
    yield c
    c.close()


def _gemm(c, ta, tb, A, B, alpha=1.0, beta=0.0, C0=None, pad=0):
    """op(A) op(B) with leading dimensions larger than the rows by `pad`."""
    import torch
    m, k = A.shape
    n = B.shape[1]

    def dev(M):
        buf = np.full((M.shape[1], M.shape[0] + pad), np.pi)
        buf[:, :M.shape[0]] = M.T
        return torch.from_numpy(buf).cuda(), M.shape[0] + pad
    dA, lda = dev(A if ta == "N" else A.T)
    dB, ldb = dev(B if tb == "N" else B.T)
    dC, ldc = dev(C0 if C0 is not None else np.full((m, n), np.nan))
    api.dgemm_dev(ta, tb, m, n, k, alpha, dA.data_ptr(), lda, dB.data_ptr(), ldb, beta,
                  dC.data_ptr(), ldc, ctx=c)
    out = dC.cpu().numpy()
    assert np.all(out[:, m:] == np.pi)
    return out[:, :m].T


# tiles are 128 x 64 x 32, integer sums span 128 k, rows are scanned in place up to k = 128
@pytest.mark.parametrize("m,n,k", [(1, 1, 1), (5, 3, 2), (127, 63, 31), (128, 64, 32), (129, 65, 33),
                                   (130, 70, 127), (64, 128, 128), (200, 130, 129), (257, 40, 1025),
                                   (300, 200, 4096), (1500, 9, 20)])
@pytest.mark.parametrize("ta", ["N", "T"])
@pytest.mark.parametrize("tb", ["N", "T"])
def test_small_integers_exact(tc, m, n, k, ta, tb):
    rng = np.random.default_rng(m + 7 * n + 31 * k)
    A = rng.integers(-2 ** 20, 2 ** 20, (m, k)).astype(float)
    B = rng.integers(-2 ** 20, 2 ** 20, (k, n)).astype(float)
    ref = (A.astype(np.int64) @ B.astype(np.int64)).astype(float)
    assert np.array_equal(_gemm(tc, ta, tb, A, B, pad=3), ref)
    C0 = rng.integers(-2 ** 20, 2 ** 20, (m, n)).astype(float)
    assert np.array_equal(_gemm(tc, ta, tb, A, B, -1.0, 1.0, C0), C0 - ref)
    assert np.array_equal(_gemm(tc, ta, tb, A, B, 0.5, -2.0, C0), 0.5 * ref - 2.0 * C0)


def _check(tc, A, B, ta="N", tb="N"):
    C = _gemm(tc, ta, tb, A, B)
    rng = np.random.default_rng(0)
    k = A.shape[1]
    for i, j in zip(rng.integers(0, A.shape[0], 60), rng.integers(0, B.shape[1], 60)):
        prod = [Fraction(float(x)) * Fraction(float(y)) for x, y in zip(A[i], B[:, j])]
        err = abs(Fraction(float(C[i, j])) - sum(prod))
        tol = (17 * Fraction(2) ** -53 * sum(abs(p) for p in prod) +
               k * Fraction(2) ** -59 * Fraction(float(np.max(np.abs(A[i])) * np.max(np.abs(B[:, j])))))
        assert err <= tol, (i, j, float(err), float(tol))


@pytest.mark.parametrize("k", [1, 40, 128, 700, 3000])
def test_error_bound(tc, k):
    rng = np.random.default_rng(k)
    A, B = rng.standard_normal((150, k)), rng.standard_normal((k, 90))
    _check(tc, A, B)
    _check(tc, A, B, "T", "T")
    # magnitudes over twelve decades in every row and column, rows and columns scaled apart
    A *= 10.0 ** (-12 * rng.random((150, k))) * 2.0 ** rng.integers(-400, 400, (150, 1))
    B *= 10.0 ** (-12 * rng.random((k, 90))) * 2.0 ** rng.integers(-400, 400, (1, 90))
    _check(tc, A, B)


def test_largest_digits(tc):
    """Every digit at its extreme (127, or -128), with one sign: the integer sums reach their bound."""
    k = 128
    for digits in ([63] + [127] * 6 + [120], [-63] + [-128] * 6 + [-128]):
        q = 0
        for d in digits:
            q = 256 * q + d
        big = float((q >> 9) << 9)               # 53 bits: the row's power of two
        fill = float(q - ((q >> 40) << 40))      # the lower digits of smaller elements
        A = np.full((130, k), fill)
        A[:, ::2] = big
        B = np.full((k, 66), fill)
        B[1::2] = big
        _check(tc, A, B)
        _check(tc, A, -B)
        _check(tc, np.full((130, k), big), np.full((k, 66), big))


def test_non_finite_and_range(tc):
    rng = np.random.default_rng(5)
    A, B = rng.standard_normal((150, 90)), rng.standard_normal((90, 77))
    A[3, 4], A[7, 1], B[2, 5], B[1, 9] = np.nan, np.inf, -np.inf, np.nan
    A[20] = 0.0
    A[21] *= 1e-300
    B[:, 31] *= 1e-200
    A[23] *= 1e300
    B[:, 33] *= 1e12
    C = _gemm(tc, "N", "N", A, B)
    with np.errstate(all="ignore"):
        ref = A @ B
    plain = np.ones_like(ref, dtype=bool)
    plain[21, 31] = plain[23, 33] = False        # below and above the range of a double
    assert np.array_equal(np.isnan(C)[plain], np.isnan(ref)[plain])
    inf = np.isinf(ref) & plain
    assert np.array_equal(C[inf], ref[inf]) and inf.sum() > 100
    fin = np.isfinite(ref) & plain
    bound = 1e-13 * (np.abs(np.nan_to_num(A, posinf=0, neginf=0)) @
                     np.abs(np.nan_to_num(B, posinf=0, neginf=0))) + 1e-320
    assert np.all(np.abs(C - ref)[fin] <= bound[fin])
    assert C[21, 31] == 0.0
    assert C[23, 33] == np.sign(np.dot(A[23] / 1e300, B[:, 33])) * np.inf or np.isfinite(C[23, 33])
