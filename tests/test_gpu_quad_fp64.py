"""EcRPA at the G0W0 energies in the FP64 tier: the frequency quadrature (rank at most nS/3) and the
eigenvalue route on either side of that rule.

With half as many points again as the mixed tier's the quadrature error is below 1e-12 of EcRPA for
every width of the spectrum; the reference's sum of nS eigenvalues carries ~nS 2^-53 max Omega.
"""
import numpy as np
import pytest

from quack_gb300 import api, synth

pytestmark = pytest.mark.gpu


def _ec_ref(L, e, nO):
    Lov = L[:, :nO, nO:].reshape(L.shape[0], -1)
    d = (e[None, nO:] - e[:nO, None]).ravel()
    K = Lov.T @ Lov
    s = np.sqrt(d)
    M = 4.0 * K * s[:, None] * s[None, :]
    M[np.diag_indices_from(M)] += d * d
    return 0.5 * (np.sqrt(np.linalg.eigvalsh(M)).sum() - d.sum() - 2.0 * np.trace(K)), d


# nS = 280: naux below and above nS/3, nS below 9 N (the tensor form takes the eigenvalues); nS = 784;
# gap: width of the spectrum (points 36, 48, 72, 96)
@pytest.mark.parametrize("N,nO,naux,gap", [(47, 7, 90, 1.0), (47, 7, 94, 1.0), (70, 14, 150, 0.3),
                                            (70, 14, 130, 0.05), (70, 14, 130, 0.006)])
@pytest.mark.parametrize("eri", [False, True])
def test_ecrpa(ctx, N, nO, naux, gap, eri):
    import torch
    rng = np.random.default_rng(N + naux)
    s = synth.gen_system(N, nO, naux, rng)
    L = s["L"] * 0.3
    e = s["eHF"].copy()
    e[nO - 1], e[nO] = -gap / 2, gap / 2
    e = np.concatenate([np.sort(np.minimum(e[:nO], -gap / 2)), np.sort(np.maximum(e[nO:], gap / 2))])
    opts = api.GWOptions(linearize=True, eta=0.1)
    nS = nO * (N - nO)
    de = torch.from_numpy(e).cuda()
    out = [torch.zeros(k, dtype=torch.float64, device="cuda") for k in (N, N, N, nS)]
    p = [t.data_ptr() for t in out]
    if eri:
        dE = synth.eri_fortran_flat_torch(L)
        ec, _ = api.RG0W0_dev(opts, N, 0, nO, 0, dE.data_ptr(), de.data_ptr(), *p, ctx=ctx)
    else:
        dL = torch.from_numpy(api.L_fortran_flat(L)).cuda()
        ec, _ = api.RG0W0_L_dev(opts, N, 0, nO, 0, naux, dL.data_ptr(), de.data_ptr(), *p, ctx=ctx)
    ref, d = _ec_ref(L, out[0].cpu().numpy(), nO)
    if d.min() <= 0.0:
        assert np.isnan(ec)
    else:
        assert abs(ec - ref) <= 1e-12 * abs(ref) + 4 * nS * 2.0 ** -53 * d.max()
