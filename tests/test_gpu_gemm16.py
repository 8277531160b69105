"""The DFMA GEMM's 16 x 16 tiles at their edges, its split of K and its one-dimensional grid.

Bound: a chain of k fused multiply-adds, the additions of the split's parts and alpha, beta:
(k + 40) 2^-53 of |alpha| |A| |B| + |beta| |C|, and as much again for numpy's product.
"""
import numpy as np
import pytest

from quack_gb300 import api

pytestmark = pytest.mark.gpu
U = 2.0 ** -53


@pytest.mark.parametrize("m,n,k", [(1, 1, 1), (15, 17, 31), (16, 16, 32), (17, 33, 33), (48, 48, 48),
                                   (129, 5, 64), (3, 200, 700), (65, 66, 1000)])
@pytest.mark.parametrize("ta,tb", [("N", "N"), ("T", "N"), ("N", "T"), ("T", "T")])
def test_dfma_tiles(ctx, m, n, k, ta, tb):
    import torch
    rng = np.random.default_rng(m * 1000 + n + k)
    lda, ldb, ldc = (m if ta == "N" else k) + 3, (k if tb == "N" else n) + 1, m + 2
    A = np.asfortranarray(rng.standard_normal((lda, k if ta == "N" else m)))
    B = np.asfortranarray(rng.standard_normal((ldb, n if tb == "N" else k)))
    C = np.asfortranarray(rng.standard_normal((ldc, n)))
    dev = [torch.from_numpy(x.ravel(order="F").copy()).cuda() for x in (A, B, C)]
    torch.cuda.synchronize()
    api.dgemm_dev(ta, tb, m, n, k, -1.5, dev[0].data_ptr(), lda, dev[1].data_ptr(), ldb, 0.75,
                  dev[2].data_ptr(), ldc, ctx=ctx)
    got = dev[2].cpu().numpy().reshape((ldc, n), order="F")
    a = A[:m, :k] if ta == "N" else A[:k, :m].T
    b = B[:k, :n] if tb == "N" else B[:n, :k].T
    ref = -1.5 * (a @ b) + 0.75 * C[:m]
    bound = 2 * (k + 40) * U * (1.5 * np.abs(a) @ np.abs(b) + 0.75 * np.abs(C[:m]))
    assert np.all(np.abs(got[:m] - ref) <= bound)
    assert np.array_equal(got[m:], C[m:])      # the rows below C stay as they were
