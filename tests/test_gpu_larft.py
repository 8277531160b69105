"""The T factors of the back-transformation at the edges of a block of 128 reflectors.

The residual A z - w z of a backward stable reduction with Householder blocks is a small multiple of
n 2^-53 ||A||_F per vector; 16 n 2^-53 is asked for.
"""
import numpy as np
import pytest

from quack_gb300 import api

pytestmark = pytest.mark.gpu
U = 2.0 ** -53


# n - 2 reflectors: none, one, 31 to 33, a block less one, full, one more, two blocks and one more
@pytest.mark.parametrize("n", [2, 3, 33, 34, 35, 129, 130, 131, 259])
@pytest.mark.parametrize("mode", [0, 1, 2])
def test_back_transformation(ctx, n, mode):
    import torch
    rng = np.random.default_rng(n)
    A = rng.standard_normal((n, n))
    A = A + A.T
    d = torch.from_numpy(A.copy()).cuda()
    w = torch.empty(n, dtype=torch.float64, device="cuda")
    Z = torch.empty(n, n, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    ctx.tune_set("dsyev_df", 0, mode)
    try:
        api.dsyev_dev(n, d.data_ptr(), n, w.data_ptr(), Z.data_ptr(), True, ctx=ctx)
    finally:
        ctx.tune_set("dsyev_df", 0, 0)
    w, Z = w.cpu().numpy(), Z.cpu().numpy()      # Z[i, j]: component i of eigenvector j
    assert np.max(np.abs(A @ Z - Z * w)) <= 16 * n * U * np.linalg.norm(A)
