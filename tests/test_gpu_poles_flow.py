"""SRG pole sums with flows that are not positive, where the weight 1 - exp(-2 s eps^2) is small, zero
or negative, at excitation counts that leave padding lanes (not a multiple of 32).
"""
import numpy as np
import pytest

from quack_gb300 import api

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("flow", [-1e-3, -0.05, 0.0, 1e-6])
@pytest.mark.parametrize("N,nO", [(9, 4), (17, 3), (12, 4)])
def test_flow(ctx, N, nO, flow):
    rng = np.random.default_rng(N)
    nS = nO * (N - nO)
    e = np.concatenate([np.sort(rng.uniform(-3, -0.3, nO)), np.sort(rng.uniform(0.05, 5, N - nO))])
    Om = np.sort(rng.uniform(0.4, 6.0, nS))
    rho = np.asfortranarray(rng.standard_normal((N, N, nS)) * 0.05)
    gm, Sig, Z = api.RGW_SRG_self_energy_diag(flow, N, N, 0, nO, N - nO, 0, nS, e, Om, rho, ctx=ctx)
    sgn = np.where(np.arange(N) < nO, 1.0, -1.0)
    eps = e[:, None, None] - e[None, :, None] + sgn[None, :, None] * Om       # [p, q, m]
    t = 2.0 * rho ** 2 * -np.expm1(-2.0 * flow * eps ** 2)
    # 1 - exp(.) carries 4 ulp of max(1, exp(.)), the rest of a term and its sums 64 ulp of it
    u = 2.0 ** -53
    w = 2.0 * rho ** 2 * (4 * u * np.maximum(1.0, np.exp(-2.0 * flow * eps ** 2))) + 80 * u * np.abs(t)
    bound = lambda a: 2 * a.sum(axis=(1, 2))
    assert np.all(np.abs(Sig - (t / eps).sum(axis=(1, 2))) <= bound(w / np.abs(eps)))
    inv = 1.0 + (t / eps ** 2).sum(axis=(1, 2))
    assert np.all(np.abs(1 / Z - inv) <= bound(w / eps ** 2) + 8 * u * (1 + np.abs(inv)))
    ref = -2.0 * (t / eps)[nO:, :nO].sum()
    assert abs(gm - ref) <= 4 * (w / np.abs(eps))[nO:, :nO].sum() + 64 * u * abs(ref)
