"""The tensor-core FP64 products in panels, as operands with more than 2 GiB of digit planes take them:
the setting "tc_panel" lowers that bound, so that every operand above one tile is cut.  Products of
small integers are exact however they are cut.
"""
import numpy as np
import pytest

from quack_gb300 import api, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k", [(128, 64, 40), (129, 65, 33), (300, 130, 129), (257, 300, 1025)])
@pytest.mark.parametrize("ta,tb", [("N", "N"), ("T", "T")])
def test_products(m, n, k, ta, tb):
    import torch
    rng = np.random.default_rng(m + n + k)
    A = rng.integers(-2 ** 20, 2 ** 20, (m, k)).astype(float)
    B = rng.integers(-2 ** 20, 2 ** 20, (k, n)).astype(float)
    dA = torch.from_numpy(np.ascontiguousarray(A.T if ta == "N" else A)).cuda()
    dB = torch.from_numpy(np.ascontiguousarray(B.T if tb == "N" else B)).cuda()
    dC = torch.full((n, m), np.nan, dtype=torch.float64, device="cuda")
    c = api.Context(0)
    try:
        for b in range(40):
            c.tune_set("dgemm_path", 2 ** b, 3)
        c.tune_set("tc_panel", 0, 1)
        api.dgemm_dev(ta, tb, m, n, k, 1.0, dA.data_ptr(), m if ta == "N" else k, dB.data_ptr(),
                      k if tb == "N" else n, 0.0, dC.data_ptr(), m, ctx=c)
    finally:
        c.close()
    ref = (A.astype(np.int64) @ B.astype(np.int64)).astype(float)
    assert np.array_equal(dC.cpu().numpy().T, ref)


# rank 150, 260: two and three panels of the quadrature's r x r products (lower triangle only)
@pytest.mark.parametrize("N,nO,naux", [(70, 14, 150), (76, 16, 260)])
def test_quadrature(N, nO, naux):
    import torch
    s = synth.gen_system(N, nO, naux, np.random.default_rng(naux))
    L = s["L"] * 0.3
    e = s["eHF"].copy()
    e[:nO] -= 0.4
    nS = nO * (N - nO)
    dL = torch.from_numpy(api.L_fortran_flat(L)).cuda()
    de = torch.from_numpy(e).cuda()
    out = [torch.zeros(k, dtype=torch.float64, device="cuda") for k in (N, N, N, nS)]
    c = api.Context(0)
    try:
        c.tune_set("tc_panel", 0, 1)
        ec, _ = api.RG0W0_L_dev(api.GWOptions(linearize=True, eta=0.1), N, 0, nO, 0, naux,
                                dL.data_ptr(), de.data_ptr(), *[t.data_ptr() for t in out], ctx=c)
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
