"""Basis functions scaled by powers of two (unnormalised functions): the orbitals' coefficients take the
inverse, every product of the AO to MO transformation and of qsGW scales exactly, and the results are
the same bits.
"""
import numpy as np
import pytest

from quack_gb300 import api, synth

pytestmark = pytest.mark.gpu


def _scales(n, rng, width):
    return 2.0 ** rng.integers(-width, width + 1, n)


def _t4(E, s):
    return E * s[:, None, None, None] * s[:, None, None] * s[:, None] * s


# 12: every product on DFMA; 40, 65: tensor cores (one and two column tiles)
@pytest.mark.parametrize("n,m", [(12, 12), (40, 40), (65, 61)])
@pytest.mark.parametrize("width", [3, 20, 45])
def test_aotomo(ctx, n, m, width):
    rng = np.random.default_rng(n)
    L = rng.standard_normal((n, n, n)) * 0.3
    L = L + L.transpose(0, 2, 1)
    E = np.einsum("Pac,Pbd->abcd", L, L, optimize=True)
    C = rng.standard_normal((n, m))
    s = _scales(n, rng, width)
    ref = api.AOtoMO_ERI_RHF(n, m, C, E, ctx=ctx)
    assert np.array_equal(api.AOtoMO_ERI_RHF(n, m, C / s[:, None], _t4(E, s), ctx=ctx), ref)
    x = np.einsum("abcd,ap,bq,cr,ds->pqrs", E, C, C, C, C, optimize=True)
    assert np.max(np.abs(ref - x)) <= 1e-12 * np.max(np.abs(x))


@pytest.mark.parametrize("zero", [False, True])
def test_aotomo_range(ctx, zero):
    """Scales at the ends of the exponent range, a function that no orbital holds, an infinity."""
    rng = np.random.default_rng(1)
    n = 40
    L = rng.standard_normal((n, n, n)) * 0.3
    L = L + L.transpose(0, 2, 1)
    E = np.einsum("Pac,Pbd->abcd", L, L, optimize=True)
    C = rng.standard_normal((n, n))
    s = np.ones(n)
    s[::2], s[1::4] = 2.0 ** 200, 2.0 ** -200
    if zero:
        C[7] = 0.0
    ref = api.AOtoMO_ERI_RHF(n, n, C, E, ctx=ctx)
    got = api.AOtoMO_ERI_RHF(n, n, C / s[:, None], _t4(E, s), ctx=ctx)
    assert np.array_equal(got, ref)
    E[3, 4, 5, 6] = np.inf
    C[3] = np.abs(C[3])
    with np.errstate(invalid="ignore"):
        assert not np.isfinite(api.AOtoMO_ERI_RHF(n, n, C, E, ctx=ctx)).any()


@pytest.mark.parametrize("width", [20])
def test_qsgw(ctx, width):
    h = synth.hchain_system(12)
    n, nO = h["nBas"], h["nO"]
    s = _scales(n, np.random.default_rng(2), width)
    o = api.GWOptions(eta=0.1, maxSCF=2)

    def run(s):
        ss = s[:, None] * s
        return api.qsRGW(o, n, n, 0, nO, n - nO, 0, nO * (n - nO), h["eHF"], h["cHF"] / s[:, None],
                         h["PHF"] / ss, h["S"] * ss, h["T"] * ss, h["V"] * ss, h["Hc"] * ss,
                         h["X"] / s[:, None], _t4(h["ERI_AO"], s), ctx=ctx, raise_on_fail=False)
    a, b = run(np.ones(n)), run(s)
    for k in ("eGW", "Z"):
        assert np.array_equal(a[k], b[k])
    assert np.array_equal(a["c"], b["c"] * s[:, None])


def test_qsgw_large():
    """One cycle of 240 functions, where products of nBas^3 would be worth the tensor cores."""
    import torch
    n, nO, naux = 240, 2, 30
    g = torch.Generator(device="cuda").manual_seed(4)
    r = lambda *k: torch.randn(*k, generator=g, device="cuda", dtype=torch.float64)
    B = r(n, n) * 0.02
    S = torch.eye(n, device="cuda", dtype=torch.float64) + B @ B.T
    w, U = torch.linalg.eigh(S)
    X = U @ torch.diag(w.rsqrt()) @ U.T
    T = torch.diag(torch.linspace(0.5, 4.0, n, device="cuda", dtype=torch.float64))
    V = r(n, n) * 0.01
    V = -(V + V.T) - torch.diag(torch.linspace(3.0, 0.1, n, device="cuda", dtype=torch.float64))
    e, Cp = torch.linalg.eigh(X.T @ (T + V) @ X)
    c = X @ Cp
    P = 2.0 * c[:, :nO] @ c[:, :nO].T
    L = r(naux, n, n) * 0.005
    L = L + L.transpose(1, 2)
    s = torch.from_numpy(_scales(n, np.random.default_rng(3), 20)).cuda()
    f = lambda x: x.T.contiguous().reshape(-1)                   # Fortran order
    Lf = L.reshape(naux, n * n)
    E = (Lf.T @ Lf).reshape(n, n, n, n).permute(3, 1, 2, 0).contiguous()
    ctx = api.Context(0)
    res = []
    try:
        for k in (torch.ones_like(s), s):
            kk = k[:, None] * k
            E.mul_(k[:, None, None, None]).mul_(k[:, None, None]).mul_(k[:, None]).mul_(k)
            ins = [e, f(c / k[:, None]), f(P / kk), f(S * kk), f(T * kk), f(V * kk), f((T + V) * kk),
                   f(X / k[:, None]), E]
            out = [torch.zeros(m, dtype=torch.float64, device="cuda") for m in (n, n * n, n * n, n)]
            api.qsRGW_dev(api.GWOptions(eta=0.1, maxSCF=0), n, 0, nO, 0, *[t.data_ptr() for t in ins],
                          *[t.data_ptr() for t in out], ctx=ctx, raise_on_fail=False)
            res.append([out[0], out[1].reshape(n, n).T * k[:, None], out[3]])
    finally:
        ctx.close()
    del E, ins, L, Lf
    torch.cuda.empty_cache()
    for a, b in zip(*res):
        assert torch.isfinite(a).all() and torch.equal(a, b)
