"""The FP64 pole sums at the edges of their tiles (8 orbitals, 32 excitations, 8 warps of q), in the
three forms (eta = 0, eta, SRG) and through both entry points, against the same sums in torch FP64.

Bound, u = 2^-53: the pole distance eps carries u (|w - e| + 2 |Om| + |eps|) on each side, which
moves a term by that times its slope; the other operations of a term and the exp add 16 u of it,
and in the SRG weight 1 - exp(.) 4 u absolutely; the sums add 64 u of the sum of magnitudes (chains
shorter than 64 additions in the kernel, pairwise sums in torch).  Twice all of it, for the two
sides.
"""
import numpy as np
import pytest

from quack_gb300 import api

pytestmark = pytest.mark.gpu
U = 2.0 ** -53


def _inputs(N, nO, nC, nR, seed):
    import torch
    g = torch.Generator(device="cuda").manual_seed(seed)
    nS = (nO - nC) * (N - nO - nR)
    r = lambda *s: torch.rand(*s, generator=g, device="cuda", dtype=torch.float64)
    e = torch.cat([torch.sort(-20 + 19.7 * r(nO)).values, torch.sort(0.05 + 5 * r(N - nO)).values])
    Om = torch.sort(0.4 + 25 * r(nS)).values
    rho = torch.randn(nS, N, N, generator=g, device="cuda", dtype=torch.float64) * 0.05
    return nS, e, Om, rho


def _reference(kind, par, N, nO, nC, nR, e, Om, rho):
    """[Sigma, dSigma, occupied part] per orbital and their bounds"""
    import torch
    q = torch.arange(N, device="cuda")
    act = ((q >= nC) & (q < N - nR)).double()
    sgn = torch.where(q < nO, 1.0, -1.0).double()
    S = torch.zeros(6, N, dtype=torch.float64, device="cuda")
    for p in range(nC, N - nR):
        x2 = 2 * rho[:, :, p] ** 2 * act                       # [m, q]
        c = e[p] - e
        eps = c[None] + sgn[None] * Om[:, None]
        de = U * (c.abs()[None] + 2 * Om[:, None] + eps.abs())
        if kind == "eta":
            d = eps ** 2 + par ** 2
            f, df = eps / d, -(eps ** 2 - par ** 2) / d ** 2
            sf, sd = 1 / d, 6 / (d * d.sqrt())                  # slopes of f and of df
            rf, rd = 16 * U * f.abs(), 16 * U / d
        else:
            s = par if kind == "srg" else np.inf
            g = 1 - torch.exp(-2 * s * eps ** 2) if kind == "srg" else torch.ones_like(eps)
            f, df = g / eps, -g / eps ** 2
            k = torch.zeros_like(eps) if kind == "eta0" else 4 * s * (1 - g)
            sf, sd = g / eps ** 2 + k, (2 * g / eps ** 2 + 2 * k) / eps.abs()
            ab = 4 * U if kind == "srg" else 0.0
            rf, rd = 16 * U * f.abs() + ab / eps.abs(), 16 * U * df.abs() + ab / eps ** 2
        S[0, p], S[1, p], S[2, p] = (x2 * f).sum(), (x2 * df).sum(), (x2 * f)[:, :nO].sum()
        S[3, p] = 2 * (x2 * (sf * de + rf + 64 * U * f.abs())).sum()
        S[4, p] = 2 * (x2 * (sd * de + rd + 64 * U * df.abs())).sum()
    return S.cpu().numpy()


def _check(N, nO, nC, nR, S, gm, Sig, Z):
    act = slice(nC, N - nR)
    assert np.all(np.abs(Sig - S[0])[act] <= S[3][act])
    # Z = 1/(1 - dSigma): the bound of dSigma on 1/Z, with the rounding of the two divisions
    inv = 1 - S[1]
    assert np.all(np.abs(1 / Z - inv)[act] <= (S[4] + 4 * U * (1 + np.abs(inv)))[act])
    assert np.all(np.delete(Sig, np.arange(nC, N - nR)) == 0.0)
    occ = slice(nO, N - nR)
    ref = -2 * S[2][occ].sum()
    assert abs(gm - ref) <= 2 * S[3][occ].sum() + 64 * U * np.abs(2 * S[2][occ]).sum()


# active orbitals 2 (a lone warp lane pair), 8, 9, 15, 17, 61 - 3; nS below, at and above 32 lanes
@pytest.mark.parametrize("N,nO,nC,nR", [(2, 1, 0, 0), (8, 4, 0, 0), (9, 5, 1, 1), (12, 4, 0, 0),
                                        (17, 3, 0, 2), (33, 1, 0, 0), (61, 9, 1, 2)])
@pytest.mark.parametrize("kind,par", [("eta0", 0.0), ("eta", 0.05), ("eta", 3.0), ("srg", 500.0),
                                      ("srg", 0.5)])
def test_pole_sums(ctx, N, nO, nC, nR, kind, par):
    nS, e, Om, rho = _inputs(N, nO, nC, nR, N)
    S = _reference(kind, par, N, nO, nC, nR, e, Om, rho)
    h = (e.cpu().numpy(), Om.cpu().numpy(), np.asfortranarray(rho.cpu().numpy().transpose(2, 1, 0)))
    fn = api.RGW_SRG_self_energy_diag if kind == "srg" else api.RGW_self_energy_diag
    gm, Sig, Z = fn(par, N, N, nC, nO, N - nO, nR, nS, *h, ctx=ctx)
    _check(N, nO, nC, nR, S, gm, Sig, Z)


# the allocation-free entry: one 32-lane group a chunk up to nS = 4096, more above
@pytest.mark.parametrize("N,nO,nC,nR", [(9, 5, 1, 1), (61, 9, 1, 2), (132, 52, 0, 0)])
@pytest.mark.parametrize("eta", [0.0, 0.05])
def test_noalloc(N, nO, nC, nR, eta):
    import torch
    nS, e, Om, rho = _inputs(N, nO, nC, nR, N)
    out = [torch.full((k,), 7.0, dtype=torch.float64, device="cuda") for k in (1, N, N)]
    torch.cuda.synchronize()
    assert api.RGW_self_energy_diag_noalloc_dev(eta, N, N, nC, nO, N - nO, nR, nS, e.data_ptr(),
                                                Om.data_ptr(), rho.data_ptr(),
                                                *[t.data_ptr() for t in out]) == 0
    S = _reference("eta" if eta else "eta0", eta, N, nO, nC, nR, e, Om, rho)
    _check(N, nO, nC, nR, S, float(out[0]), out[1].cpu().numpy(), out[2].cpu().numpy())
