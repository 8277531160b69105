"""The fixed-point tridiagonalisation of the FP64 tier's drivers, through qk_dsyev_dev with the
context setting dsyev_df = 2.

An element update rounds to 2^-62 S with S < 4 ||A||_F, so over n columns the backward error of an
eigenvalue is far below n 2^-53 ||A||_F, the bound used here; the eigenvectors' residuals carry the
inverse iteration and the back-transformation as well (8 times that).  Sizes: every cluster size,
their edges, the largest matrix of the cluster form (615) and sizes of the grid form, where the
number of CTAs must not change a bit.
"""
import numpy as np
import pytest

from quack_gb300 import api

pytestmark = pytest.mark.gpu
SIZES = [2, 3, 31, 33, 64, 65, 128, 129, 257, 615, 616, 801]


def _eig(c, A, lower_only=False):
    import torch
    n = A.shape[0]
    M = np.where(np.tri(n, dtype=bool), A, np.nan) if lower_only else A
    dA = torch.from_numpy(np.ascontiguousarray(M.T)).cuda()
    w = torch.empty(n, dtype=torch.float64, device="cuda")
    Z = torch.empty(n, n, dtype=torch.float64, device="cuda")
    api.dsyev_dev(n, dA.data_ptr(), n, w.data_ptr(), Z.data_ptr(), True, ctx=c)
    return w.cpu().numpy(), Z.cpu().numpy()          # Z[i, j]: component i of eigenvector j


@pytest.fixture()
def fx():
    c = api.Context(0)
    c.tune_set("dsyev_df", 0, 2)
    yield c
    c.close()


def _casida(n, rng):
    d = np.sort(rng.uniform(0.35, 25.0, n))
    K = rng.standard_normal((n, n // 3 + 4)) * 0.05
    s = np.sqrt(d)
    return 4.0 * (K @ K.T) * np.outer(s, s) + np.diag(d * d)


def _check(c, A):
    n = A.shape[0]
    w, Z = _eig(c, A, lower_only=True)
    fro = np.linalg.norm(A)
    ref = np.linalg.eigvalsh(A)
    assert np.max(np.abs(w - ref)) <= n * 2.0 ** -53 * fro
    assert np.max(np.abs(A @ Z - Z * w)) <= 8 * n * 2.0 ** -53 * fro
    assert np.max(np.abs(Z.T @ Z - np.eye(n))) <= 1e-10
    w2, Z2 = _eig(c, A)
    assert np.array_equal(w, w2) and np.array_equal(Z, Z2)


@pytest.mark.parametrize("n", SIZES)
def test_casida_and_dense(fx, n):
    rng = np.random.default_rng(n)
    _check(fx, _casida(n, rng))
    A = rng.standard_normal((n, n))
    _check(fx, A + A.T)


@pytest.mark.parametrize("n", [33, 300, 640])
def test_degenerate_columns(fx, n):
    """Columns already reduced, columns of tiny norm, rank deficiency, extreme magnitudes."""
    rng = np.random.default_rng(n)
    x = rng.standard_normal((n, 3))
    _check(fx, x @ x.T)
    T = np.diag(rng.standard_normal(n)) + np.diag(rng.standard_normal(n - 1), 1)
    _check(fx, T + T.T)
    A = np.diag(rng.uniform(1.0, 2.0, n))
    A[:n // 2, n // 2:] = 1e-9 * rng.standard_normal((n // 2, n - n // 2))
    _check(fx, np.tril(A.T) + np.tril(A.T, -1).T)
    C = _casida(n, rng)
    for scale in (2.0 ** 300, 2.0 ** -300):
        w, _ = _eig(fx, C * scale)
        assert np.array_equal(w, _eig(fx, C)[0] * scale)


@pytest.mark.parametrize("n", [50, 650])
def test_nan_gives_nan(fx, n):
    A = _casida(n, np.random.default_rng(1))
    A[20, 7] = A[7, 20] = np.nan
    assert np.isnan(_eig(fx, A)[0]).all()


def test_grid_form_independent_of_the_cta_count(fx):
    A = _casida(700, np.random.default_rng(3))
    outs = []
    for quarters in (4, 1, 3):
        fx.tune_set("sytrd_grid", 700, quarters)
        outs.append(_eig(fx, A))
    for w, Z in outs[1:]:
        assert np.array_equal(w, outs[0][0]) and np.array_equal(Z, outs[0][1])
