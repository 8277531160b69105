"""The attempt at a factor of (ia|jb) for EcRPA in the FP64 tier: given up after N pivots for the
integrals of hydrogen chains, whose rank is about 5 N, and carried through for a tensor of 2 N or 3 N factors.
The energy is that of the Casida eigenvalues either way.
"""
import numpy as np
import pytest

from quack_gb300 import api, synth

pytestmark = pytest.mark.gpu


def _run(ctx, T, e, N, nO):
    import torch
    de = torch.from_numpy(np.ascontiguousarray(e)).cuda()
    out = [torch.zeros(k, dtype=torch.float64, device="cuda") for k in (N, N, N, nO * (N - nO))]
    ec, _ = api.RG0W0_dev(api.GWOptions(linearize=True, eta=0.1), N, 0, nO, 0, T.data_ptr(),
                          de.data_ptr(), *[t.data_ptr() for t in out], ctx=ctx)
    E = T.reshape(N, N, N, N).cpu().numpy()                      # [s, r, q, p] of <pq|rs>
    K = E[nO:, :nO, :nO, nO:].transpose(2, 0, 1, 3).reshape(nO * (N - nO), -1)   # (ia|jb) = <ij|ab>
    eGW = out[0].cpu().numpy()
    d = (eGW[None, nO:] - eGW[:nO, None]).ravel()
    assert d.min() > 0.0
    q = np.sqrt(d)
    M = 4.0 * 0.5 * (K + K.T) * q[:, None] * q[None, :]
    M[np.diag_indices_from(M)] += d * d
    w = np.linalg.eigvalsh(M)
    ref = 0.5 * (np.sqrt(w).sum() - d.sum() - 2.0 * np.trace(K))
    # the tensor's transformation leaves (ia|jb) unsymmetric by its rounding, read once on each side
    asym = np.abs(K - K.T).max()
    assert abs(ec - ref) <= 1e-12 * abs(ref) + 4 * len(d) * (2.0 ** -53 * np.sqrt(w[-1]) + asym)
    return ctx.tune_query("quad_pivots", 0)


@pytest.mark.parametrize("atoms", [24, 28])
def test_hydrogen_chain(ctx, atoms):
    import torch
    h = synth.hchain_system(atoms)
    N, nO = h["nBas"], h["nO"]
    assert nO * (N - nO) >= 9 * N
    C = torch.from_numpy(np.ascontiguousarray(h["cHF"].T)).cuda()
    E = torch.from_numpy(np.asarray(h["ERI_AO"]).ravel(order="F").copy()).cuda()
    T = torch.zeros_like(E)
    api.AOtoMO_ERI_RHF_dev(N, N, C.data_ptr(), E.data_ptr(), T.data_ptr(), ctx=ctx)
    assert _run(ctx, T, h["eHF"], N, nO) == N


@pytest.mark.parametrize("N,nO,naux", [(70, 14, 140), (70, 14, 210)])
def test_factors(ctx, N, nO, naux):
    s = synth.gen_system(N, nO, naux, np.random.default_rng(naux))
    e = s["eHF"].copy()
    e[:nO] -= 0.4
    T = synth.eri_fortran_flat_torch(s["L"] * 0.3)
    assert naux <= _run(ctx, T, e, N, nO) < nO * (N - nO) // 3
