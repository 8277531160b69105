"""The FP64 bisection with secant predictions, through qk_dsyev_dev on tridiagonal matrices: every
lane count (by size), clusters, multiple and graded eigenvalues.

A matrix that is already tridiagonal passes the reduction with rounding of n 2^-53 ||T|| at most;
the counts close each eigenvalue to 2^-51 relative, so n 2^-51 ||T|| bounds the error.
"""
import numpy as np
import pytest

from quack_gb300 import api

pytestmark = pytest.mark.gpu


def _w(ctx, d, e):
    import torch
    n = len(d)
    A = torch.zeros(n, n, dtype=torch.float64, device="cuda")
    A.diagonal().copy_(torch.from_numpy(np.asarray(d, dtype=float)))
    if n > 1:
        A.diagonal(1).copy_(torch.from_numpy(np.asarray(e, dtype=float)))
        A.diagonal(-1).copy_(torch.from_numpy(np.asarray(e, dtype=float)))
    w = torch.empty(n, dtype=torch.float64, device="cuda")
    api.dsyev_dev(n, A.data_ptr(), n, w.data_ptr(), 0, False, ctx=ctx)
    return w.cpu().numpy()


# 32 lanes up to n = 912 on 152 SMs, 16 up to 1824, 8 up to 3648, then 4; no grid below 256
@pytest.mark.parametrize("n", [1, 2, 33, 255, 256, 912, 913, 1825, 3700])
def test_toeplitz(ctx, n):
    w = _w(ctx, np.full(n, 2.0), np.full(n - 1, -1.0))
    ref = 2.0 - 2.0 * np.cos(np.arange(1, n + 1) * np.pi / (n + 1))
    assert np.max(np.abs(w - ref)) <= n * 2.0 ** -51 * 4.0


@pytest.mark.parametrize("kind", ["wilkinson", "glued", "equal", "graded", "zero blocks"])
@pytest.mark.parametrize("n", [63, 301])
def test_clusters(ctx, kind, n):
    rng = np.random.default_rng(n)
    d, e = np.abs(np.arange(n) - n // 2).astype(float), np.ones(n - 1)
    if kind == "glued":
        d = np.tile(np.abs(np.arange(21) - 10.0), n // 21 + 1)[:n]
        e[20::21] = 1e-9
    if kind == "equal":
        d, e = np.full(n, 3.0), np.zeros(n - 1)
    if kind == "graded":
        d = 10.0 ** -np.linspace(0, 14, n)
        e = 0.1 * np.sqrt(d[1:] * d[:-1])
    if kind == "zero blocks":
        d = rng.standard_normal(n)
        e[::3] = 0.0
    w = _w(ctx, d, e)
    ref = np.linalg.eigvalsh(np.diag(d) + np.diag(e, 1) + np.diag(e, -1))
    nrm = np.max(np.abs(ref))
    assert np.all(np.diff(w) >= 0.0)
    assert np.max(np.abs(w - ref)) <= n * 2.0 ** -51 * nrm
