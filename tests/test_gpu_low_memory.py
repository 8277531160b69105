"""Calls that run out of device memory where the tensor-core products or the quadrature of EcRPA would
want more: they go on without (the n-th allocation is made to fail), as the FMA products and the
eigenvalues need none of it.
"""
import numpy as np
import pytest

from quack_gb300 import api, synth

pytestmark = pytest.mark.gpu


# allocations 1 and 2 hold the tensors, the rest the exponents, digit planes and row maxima
@pytest.mark.parametrize("nth", [3, 4, 5, 6])
def test_aotomo(nth):
    rng = np.random.default_rng(nth)
    import torch
    n = 40
    E = rng.standard_normal((n,) * 4)
    C = rng.standard_normal((n, n))
    dE = torch.from_numpy(E.ravel(order="F").copy()).cuda()
    dC = torch.from_numpy(C.ravel(order="F").copy()).cuda()
    out = torch.zeros(n ** 4, dtype=torch.float64, device="cuda")
    c = api.Context(0)
    try:
        c.tune_set("fail_alloc", 0, nth)
        api.AOtoMO_ERI_RHF_dev(n, n, dC.data_ptr(), dE.data_ptr(), out.data_ptr(), ctx=c)
    finally:
        c.close()
    got = out.cpu().numpy().reshape((n,) * 4, order="F")
    ref = np.einsum("abcd,ap,bq,cr,ds->pqrs", E, C, C, C, C, optimize=True)
    # four contractions of n terms, each rounded n 2^-53 of the sum of magnitudes
    mag = np.einsum("abcd,ap,bq,cr,ds->pqrs", np.abs(E), *[np.abs(C)] * 4, optimize=True)
    assert np.all(np.abs(got - ref) <= 8 * n * 2.0 ** -53 * mag)


# the first G0W0 (rank above nS/3) sizes everything but the quadrature's workspace
@pytest.mark.parametrize("nth", [1, 2, 3, 4, 5, 6, 7])
def test_quadrature(nth):
    import torch
    N, nO, naux = 70, 14, 150
    nS = nO * (N - nO)
    c = api.Context(0)
    try:
        for k, fail in ((270, 0), (naux, nth)):
            s = synth.gen_system(N, nO, k, np.random.default_rng(k))
            L = s["L"] * 0.3
            e = s["eHF"].copy()
            e[:nO] -= 0.4
            dL = torch.from_numpy(api.L_fortran_flat(L)).cuda()
            de = torch.from_numpy(e).cuda()
            out = [torch.zeros(x, dtype=torch.float64, device="cuda") for x in (N, N, N, nS)]
            c.tune_set("fail_alloc", 0, fail)
            ec, _ = api.RG0W0_L_dev(api.GWOptions(linearize=True, eta=0.1), N, 0, nO, 0, k, dL.data_ptr(),
                                    de.data_ptr(), *[t.data_ptr() for t in out], ctx=c)
    finally:
        c.close()
    eGW = out[0].cpu().numpy()
    d = (eGW[None, nO:] - eGW[:nO, None]).ravel()
    assert d.min() > 0.0
    Lov = L[:, :nO, nO:].reshape(naux, -1)
    K = Lov.T @ Lov
    q = np.sqrt(d)
    M = 4.0 * K * q[:, None] * q[None, :]
    M[np.diag_indices_from(M)] += d * d
    ref = 0.5 * (np.sqrt(np.linalg.eigvalsh(M)).sum() - d.sum() - 2.0 * np.trace(K))
    assert abs(ec - ref) <= 1e-12 * abs(ref) + 4 * nS * 2.0 ** -53 * d.max()
