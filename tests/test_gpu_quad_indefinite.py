"""EcRPA at the G0W0 energies in the FP64 tier for integrals whose (ia|jb) is not positive semidefinite:
a tensor with one negative factor, and one with a single altered element (the 8 of its symmetry).  The
energy is that of the Casida eigenvalues; bound as for the semidefinite case, nS 2^-53 max Omega and
1e-12 of EcRPA.
"""
import numpy as np
import pytest

from quack_gb300 import api, synth

pytestmark = pytest.mark.gpu
N, NO, NAUX = 70, 14, 150          # nS = 784: rank 150 is below nS/3 and nS above 9 N


def _g0w0(ctx, chem, e):
    import torch
    T = torch.from_numpy(chem).cuda().permute(3, 1, 2, 0).contiguous().reshape(-1)
    de = torch.from_numpy(e).cuda()
    out = [torch.zeros(k, dtype=torch.float64, device="cuda") for k in (N, N, N, NO * (N - NO))]
    ec, _ = api.RG0W0_dev(api.GWOptions(linearize=True, eta=0.1), N, 0, NO, 0, T.data_ptr(),
                          de.data_ptr(), *[t.data_ptr() for t in out], ctx=ctx)
    return ec, out[0].cpu().numpy()


@pytest.mark.parametrize("kind", ["factor", "element"])
@pytest.mark.parametrize("size", [1.0, 0.1])
def test_indefinite(ctx, kind, size):
    rng = np.random.default_rng(3)
    s = synth.gen_system(N, NO, NAUX, rng)
    L = (s["L"] * 0.3).reshape(NAUX, N * N)
    e = s["eHF"].copy()
    e[:NO] -= 0.4
    chem = (L.T @ L).reshape(N, N, N, N)
    if kind == "factor":
        g = rng.standard_normal((N, N)) * 1e-3 * size
        g = g + g.T
        chem -= g[:, :, None, None] * g
    else:
        i, a, j, b = 2, NO + 5, 9, NO + 30
        for p, q in ((i, a), (a, i)):
            for r, t in ((j, b), (b, j)):
                chem[p, q, r, t] += 1e-3 * size
                chem[r, t, p, q] += 1e-3 * size
    K = chem[:NO, NO:, :NO, NO:].reshape(NO * (N - NO), -1)
    assert np.linalg.eigvalsh(K)[0] < -1e-6 * size
    ec, eGW = _g0w0(ctx, chem, e)
    d = (eGW[None, NO:] - eGW[:NO, None]).ravel()
    assert d.min() > 0.0
    q = np.sqrt(d)
    M = 4.0 * K * q[:, None] * q[None, :]
    M[np.diag_indices_from(M)] += d * d
    w = np.linalg.eigvalsh(M)
    assert w[0] > 0.0
    ref = 0.5 * (np.sqrt(w).sum() - d.sum() - 2.0 * np.trace(K))
    assert abs(ec - ref) <= 1e-12 * abs(ref) + 4 * len(d) * 2.0 ** -53 * np.sqrt(w[-1])
