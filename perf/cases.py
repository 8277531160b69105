"""Performance cases: what users of this framework have it compute, through its public entry points.

Every case is a dict of plain values; ``kind`` says which entry point it goes through:

  host    RG0W0 on host arrays, the drop-in for the Fortran call
  g0w0    RG0W0_dev on the MO integral tensor in device memory
  g0w0_L  RG0W0_L_dev on factorised integrals
  evgw_L  evRGW_L_dev, eigenvalue self-consistency
  batch   gw_batch_L_dev, many molecules of uneven size in one call
  bse     RGW_phBSE_dev, singlet and triplet excitation energies
  qsgw    qsRGW_dev on a hydrogen chain, a fixed number of cycles
  aomo    AOtoMO_ERI_RHF_dev, the four-index transformation
  sigma   RGW_self_energy_diag_noalloc_dev, one self-energy evaluation on caller-owned buffers

The synthetic systems have the shapes and distributions of quack_gb300.synth.gen_system (factor
entries N(0,1) * coupling / sqrt(naux), occupied levels in [-20, -0.3], virtual ones in [0.05, 5]).
``coupling`` is 0.5 there; the FP64 cases use a weaker one, which keeps the quasiparticle gap open as
in a molecule, and a finite broadening ``eta``, so that a quasiparticle energy is a smooth function
of the input.  ``mixed`` selects the mixed-precision tier.
"""
import math

import numpy as np
import torch

from quack_gb300 import api, synth

DEV = "cuda"
F64 = torch.float64


def listed():
    return [
        # the smallest call: a small molecule handed over from the Fortran host, launches and copies
        dict(name="host_n16", kind="host", N=16, nC=0, nO=4, nR=0, eta=0.05, coupling=0.2),
        # an odd-sized molecule with frozen core and virtual orbitals, linearised
        dict(name="g0w0_n61_frozen", kind="g0w0", N=61, nC=1, nO=9, nR=2, eta=0.05, coupling=0.2,
             reg=False, linearize=True, mixed=False),
        # an ordinary molecule, SRG-regularised
        dict(name="g0w0_n120_srg", kind="g0w0", N=120, nC=0, nO=15, nR=0, eta=0.0, coupling=0.2,
             reg=True, linearize=False, mixed=False),
        # the benchmark's size in the default (FP64) tier: the largest case
        dict(name="g0w0_n200", kind="g0w0", N=200, nC=0, nO=20, nR=0, eta=0.05, coupling=0.2,
             reg=False, linearize=False, mixed=False),
        # the benchmark's workload: the mixed tier with the default options (eta = 0, Newton)
        dict(name="g0w0_n200_mixed", kind="g0w0", N=200, nC=0, nO=20, nR=0, eta=0.0, coupling=0.5,
             reg=False, linearize=False, mixed=True),
        # factorised integrals, linearised quasiparticle equation
        dict(name="g0w0_L_n160", kind="g0w0_L", N=160, nC=0, nO=20, nR=0, naux=480, eta=0.05,
             coupling=0.2, linearize=True),
        # eigenvalue self-consistency: several screening problems in a row
        dict(name="evgw_L_n72", kind="evgw_L", N=72, nC=0, nO=9, nR=0, naux=216, eta=0.05,
             coupling=0.2, maxSCF=4),
        # a set of molecules of uneven size
        dict(name="batch_24", kind="batch", nsys=24, Nmin=24, Nmax=128, eta=0.05, coupling=0.2),
        # optical excitations of a small molecule
        dict(name="bse_n64", kind="bse", N=64, nC=0, nO=8, nR=0, eta=0.05, coupling=0.2),
        # quasiparticle self-consistency of H16 in 48 basis functions, three cycles
        dict(name="qsgw_h16", kind="qsgw", atoms=16, eta=0.05, maxSCF=3),
        # integral transformation with fewer orbitals than basis functions
        dict(name="aomo_n96", kind="aomo", nBas=96, nOrb=91),
        # one self-energy evaluation inside a host program's own cycle
        dict(name="sigma_n150", kind="sigma", N=150, nO=19, eta=0.05),
    ]


def _log_int(rng, a, b):
    return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))


def draw(rng):
    kind = rng.choice(["host", "g0w0", "g0w0", "g0w0", "mixed", "g0w0_L", "evgw_L", "batch", "bse",
                       "qsgw", "aomo", "sigma"])
    eta = rng.choice([0.04, 0.05, 0.07, 0.1])
    coupling = rng.choice([0.15, 0.2])
    if kind == "host":
        N = _log_int(rng, 8, 40)
        return dict(kind="host", N=N, nC=0, nO=max(2, N // rng.choice([4, 6])), nR=0, eta=eta,
                    coupling=coupling)
    if kind == "mixed":
        N = rng.randint(90, 200)
        return dict(kind="g0w0", N=N, nC=0, nO=max(4, N // 10), nR=0, eta=0.0, coupling=0.5,
                    reg=False, linearize=False, mixed=True)
    if kind == "g0w0":
        N = _log_int(rng, 30, 190)
        reg, frozen = rng.random() < 0.25, rng.random() < 0.35
        return dict(kind="g0w0", N=N, nC=int(frozen), nO=max(4, N // rng.choice([8, 10])),
                    nR=3 * frozen, eta=0.0 if reg else eta, coupling=coupling, reg=reg,
                    linearize=frozen, mixed=False)
    if kind == "g0w0_L":
        N = _log_int(rng, 40, 180)
        return dict(kind="g0w0_L", N=N, nC=0, nO=N // 8, nR=0, naux=rng.randint(2 * N, 4 * N),
                    eta=eta, coupling=coupling, linearize=rng.random() < 0.5)
    if kind == "evgw_L":
        N = _log_int(rng, 24, 110)
        return dict(kind="evgw_L", N=N, nC=0, nO=N // 8, nR=0, naux=rng.randint(2 * N, 4 * N),
                    eta=eta, coupling=coupling, maxSCF=rng.randint(2, 5))
    if kind == "batch":
        return dict(kind="batch", nsys=rng.randint(8, 32), Nmin=rng.randint(16, 40),
                    Nmax=rng.randint(60, 128), eta=eta, coupling=coupling)
    if kind == "bse":
        N = _log_int(rng, 24, 90)
        return dict(kind="bse", N=N, nC=0, nO=N // 8, nR=0, eta=eta, coupling=coupling)
    if kind == "qsgw":
        return dict(kind="qsgw", atoms=2 * rng.randint(3, 8), eta=eta, maxSCF=rng.randint(2, 4))
    if kind == "aomo":
        n = _log_int(rng, 24, 130)
        return dict(kind="aomo", nBas=n, nOrb=n - rng.randint(0, 5))
    N = _log_int(rng, 40, 200)
    return dict(kind="sigma", N=N, nO=max(4, N // rng.choice([8, 10])), eta=eta)


# ---- inputs ----------------------------------------------------------------------------------
def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    return g


def _factor(N, naux, coupling, g):
    """L[P, q, p] (symmetric in p, q): Fortran L(p, q, P)."""
    L = torch.randn(naux, N, N, generator=g, device=DEV, dtype=F64) * (coupling / math.sqrt(naux))
    up = torch.triu(L)
    return up + torch.triu(L, 1).transpose(1, 2)


def _energies(N, nO, g):
    u = torch.rand(N, generator=g, device=DEV, dtype=F64)
    occ = torch.sort(-20.0 + 19.7 * u[:nO]).values
    vir = torch.sort(0.05 + 4.95 * u[nO:]).values
    return torch.cat([occ, vir])


def _system(c, seed):
    g = _gen(seed)
    L = _factor(c["N"], c.get("naux", 3 * c["N"]), c["coupling"], g)
    return L, _energies(c["N"], c["nO"], g)


def _eri(L):
    """ERI(p,q,r,s) = <pq|rs> = (pr|qs) in Fortran order, from the factor."""
    naux, N, _ = L.shape
    Lf = L.reshape(naux, N * N)
    chem = (Lf.T @ Lf).reshape(N, N, N, N)
    return chem.permute(3, 1, 2, 0).contiguous().reshape(-1)


def _batch_systems(c, seed):
    r = np.random.default_rng([c["nsys"], c["Nmin"], c["Nmax"]])  # the sizes belong to the case
    g = _gen(seed)
    out = []
    for N in r.integers(c["Nmin"], c["Nmax"] + 1, size=c["nsys"]):
        N = int(N)
        nO = synth.n_occ(N)
        out.append((N, nO, _factor(N, 3 * N, c["coupling"], g), _energies(N, nO, g)))
    return out


def _chain(c, seed):
    spacing = 1.5 + 0.3 * np.random.default_rng(seed).random()
    return synth.hchain_system(c["atoms"], spacing)


def _aomo_inputs(c, seed):
    g = _gen(seed)
    n, m = c["nBas"], c["nOrb"]
    coef = torch.randn(m, n, generator=g, device=DEV, dtype=F64) / math.sqrt(n)  # Fortran c(mu, p)
    L = _factor(n, n, 0.5, g)
    return coef, _eri(L)


def _sigma_inputs(c, seed):
    g = _gen(seed)
    N, nO = c["N"], c["nO"]
    nS = nO * (N - nO)
    e = _energies(N, nO, g)
    d = (e[None, nO:] - e[:nO, None]).reshape(-1)
    Om = torch.sort(d + 0.3 * torch.rand(nS, generator=g, device=DEV, dtype=F64)).values
    rho = torch.randn(nS, N, N, generator=g, device=DEV, dtype=F64) * (0.2 / math.sqrt(N))
    return e, Om, rho


def _opts(c):
    return api.GWOptions(eta=c["eta"], linearize=bool(c.get("linearize", False)),
                         reg=bool(c.get("reg", False)), maxSCF=c.get("maxSCF", 64),
                         precision=api.QK_PREC_BF16X3 if c.get("mixed") else api.QK_PREC_FP64)


def _empty(*n):
    return [torch.zeros(k, dtype=F64, device=DEV) for k in n]


def prepare(case, seed):
    c = dict(case)
    kind = c["kind"]
    s = dict(c=c, ctx=api.default_context())
    if kind in ("host", "g0w0", "g0w0_L", "evgw_L", "bse"):
        N = c["N"]
        nS = (c["nO"] - c["nC"]) * (N - c["nO"] - c["nR"])
        L, e = _system(c, seed)
        s.update(nS=nS, e=e)
        if kind == "host":
            s["ERI"] = _eri(L).cpu().numpy().reshape((N,) * 4, order="F")
            s["e"] = e.cpu().numpy()
        elif kind in ("g0w0", "bse"):
            s["ERI"] = _eri(L)
        else:
            s["L"] = L
        if kind == "bse":
            s["eGW"] = torch.cat([e[:c["nO"]] - 0.05, e[c["nO"]:] + 0.05])
            s["out"] = _empty(nS, nS)
        elif kind != "host":
            s["out"] = _empty(N, N, N, nS)
        if kind != "bse":
            s["opts"] = _opts(c)
    elif kind == "batch":
        systems = _batch_systems(c, seed)
        desc = (api.qk_sys_desc * len(systems))()
        oL = oE = 0
        for i, (N, nO, L, e) in enumerate(systems):
            desc[i] = api.qk_sys_desc(N, 0, nO, 0, L.shape[0], oL, oE)
            oL += L.numel()
            oE += N
        s.update(desc=desc, L=torch.cat([x[2].reshape(-1) for x in systems]),
                 e=torch.cat([x[3] for x in systems]), opts=_opts(c))
        s["out"] = _empty(s["e"].numel())
    elif kind == "qsgw":
        h = _chain(c, seed)
        keys = ("eHF", "cHF", "PHF", "S", "T", "V", "Hc", "X", "ERI_AO")
        s["in"] = [torch.from_numpy(np.asarray(h[k]).ravel(order="F").copy()).to(DEV) for k in keys]
        n = h["nBas"]
        s.update(n=n, nO=h["nO"], opts=_opts(c), out=_empty(n, n * n, n * n, n))
    elif kind == "aomo":
        s["coef"], s["ERI"] = _aomo_inputs(c, seed)
        s["out"] = _empty(c["nOrb"] ** 4)
    else:
        s["e"], s["Om"], s["rho"] = _sigma_inputs(c, seed)
        s["out"] = _empty(1, c["N"], c["N"])
    return s


def run(s):
    c, ctx = s["c"], s["ctx"]
    kind = c["kind"]
    p = [t.data_ptr() for t in s["out"]] if "out" in s else []
    if kind == "host":
        N = c["N"]
        r = api.RG0W0(s["opts"], N, N, c["nC"], c["nO"], N - c["nO"], c["nR"], s["nS"], s["ERI"],
                      s["e"], ctx=ctx)
        return [r[k] for k in ("eGW", "SigC", "Z", "Om", "EcRPA", "EcGM")]
    if kind == "g0w0":
        ec, gm = api.RG0W0_dev(s["opts"], c["N"], c["nC"], c["nO"], c["nR"], s["ERI"].data_ptr(),
                               s["e"].data_ptr(), *p, ctx=ctx)
        return s["out"] + [ec, gm]
    if kind == "g0w0_L":
        ec, gm = api.RG0W0_L_dev(s["opts"], c["N"], c["nC"], c["nO"], c["nR"], c["naux"],
                                 s["L"].data_ptr(), s["e"].data_ptr(), *p, ctx=ctx)
        return s["out"] + [ec, gm]
    if kind == "evgw_L":
        r = api.evRGW_L_dev(s["opts"], c["N"], c["nC"], c["nO"], c["nR"], c["naux"],
                            s["L"].data_ptr(), s["e"].data_ptr(), *p[:3], ctx=ctx,
                            raise_on_fail=False)
        return s["out"][:3] + [r["EcRPA"], r["EcGM"], r["nSCF"]]
    if kind == "batch":
        r = api.gw_batch_L_dev(s["opts"], 0, s["desc"], s["L"].data_ptr(), s["e"].data_ptr(), p[0],
                               ctx=ctx)
        return [s["out"][0], r["EcRPA"], r["status"]]
    if kind == "bse":
        ec = api.RGW_phBSE_dev(api.BSEOptions(eta=c["eta"]), c["N"], c["nC"], c["nO"], c["nR"],
                               s["ERI"].data_ptr(), s["e"].data_ptr(), s["eGW"].data_ptr(), p[0],
                               p[1], ctx=ctx)
        return s["out"] + ec
    if kind == "qsgw":
        r = api.qsRGW_dev(s["opts"], s["n"], 0, s["nO"], 0, *[t.data_ptr() for t in s["in"]], p[0],
                          p[1], p[2], p[3], ctx=ctx, raise_on_fail=False)
        # the orbitals' signs are arbitrary: the density P stands for them
        return [s["out"][0], s["out"][2], s["out"][3], r["EqsGW"], r["EcRPA"], r["EcGM"], r["nSCF"]]
    if kind == "aomo":
        api.AOtoMO_ERI_RHF_dev(c["nBas"], c["nOrb"], s["coef"].data_ptr(), s["ERI"].data_ptr(), p[0],
                               ctx=ctx)
        return s["out"]
    N, nO = c["N"], c["nO"]
    rc = api.RGW_self_energy_diag_noalloc_dev(c["eta"], N, N, 0, nO, N - nO, 0, nO * (N - nO),
                                              s["e"].data_ptr(), s["Om"].data_ptr(),
                                              s["rho"].data_ptr(), *p)
    return s["out"] + [rc]


# ---- work ------------------------------------------------------------------------------------
def _gw_flops(N, nS, naux=0):
    """One G0W0: the reduction to tridiagonal form (4/3 nS^3), the excitation densities (through
    the factor where there is one) and one sweep over the pole terms."""
    rho = 2 * nS * nS * naux + 2 * N * N * nS * naux if naux else 2 * nS ** 3 + 2 * N * N * nS * nS
    return 4 / 3 * nS ** 3 + rho + 10 * N * N * nS


def work(case):
    c = dict(case)
    kind = c["kind"]
    if kind == "batch":
        Ns = np.linspace(c["Nmin"], c["Nmax"], c["nsys"])
        nS = Ns / 8 * Ns * 7 / 8
        return dict(bytes=float(np.sum(24 * Ns ** 3)),
                    flops=float(sum(_gw_flops(n, s, 3 * n) for n, s in zip(Ns, nS))))
    if kind == "qsgw":
        n, no = 3 * c["atoms"], c["atoms"] // 2
        nS = no * (n - no)
        cyc = 4 * n ** 4 * no + 4 * n ** 3 * no * (n - no) + _gw_flops(n, nS) + 2 * n ** 3 * nS
        return dict(bytes=8.0 * n ** 4, flops=float((c["maxSCF"] + 1) * cyc))
    if kind == "aomo":
        n, m = c["nBas"], c["nOrb"]
        return dict(bytes=8.0 * (n ** 4 + m ** 4),
                    flops=float(sum(2 * n ** (4 - k) * m ** (k + 1) for k in range(4))))
    if kind == "sigma":
        N, nO = c["N"], c["nO"]
        nS = nO * (N - nO)
        return dict(bytes=8.0 * N * N * nS, flops=10.0 * N * N * nS)
    N = c["N"]
    no, nv = c["nO"] - c["nC"], N - c["nO"] - c["nR"]
    nS = no * nv
    if kind in ("host", "g0w0"):
        return dict(bytes=8.0 * N * N * nS, flops=float(_gw_flops(N, nS) + 4 / 3 * nS ** 3))
    if kind == "g0w0_L":
        return dict(bytes=8.0 * N * N * c["naux"],
                    flops=float(_gw_flops(N, nS, c["naux"]) + 4 / 3 * nS ** 3))
    if kind == "evgw_L":
        return dict(bytes=8.0 * N * N * c["naux"],
                    flops=float((c["maxSCF"] + 1) * _gw_flops(N, nS, c["naux"])))
    rho = 2 * nS * nS * (no * no + nv * nv + no * nv)
    return dict(bytes=8.0 * N * N * nS,
                flops=float(rho + 4 * no * no * nv * nv * nS + 5 * 4 / 3 * nS ** 3 + 12 * nS ** 3))


# ---- the same results in plain 64-bit torch --------------------------------------------------
def _x_screening(L, e, nC, nO, nR):
    """(Om, XpY rows, tr A) of the dRPA singlet screening at energies e."""
    N = e.numel()
    Lov = L[:, nC:nO, nO:N - nR].reshape(L.shape[0], -1)
    K = Lov.T @ Lov
    d = (e[None, nO:N - nR] - e[nC:nO, None]).reshape(-1)
    sq = d.sqrt()
    M = 4.0 * K * sq[:, None] * sq[None, :]
    M.diagonal().add_(d * d)
    w, Z = torch.linalg.eigh(M)
    Om = w.abs().sqrt()
    return Om, Z.T * sq[None, :] / Om.sqrt()[:, None], float((d + 2.0 * K.diagonal()).sum()), Lov


def _x_rho(L, Lov, XpY):
    """rho[m, p, q] = sum_jb (pq|jb) XpY(m, jb)."""
    naux, N, _ = L.shape
    T = XpY @ Lov.T
    return (T @ L.reshape(naux, N * N)).reshape(-1, N, N)


def _x_poles(e, w, Om, rho, nC, nO, nR, p, eta, srg):
    """(Sigma, dSigma) of orbital p at frequency w, poles at the energies e."""
    N = e.numel()
    sig = dsig = 0.0
    for lo, hi, sgn in ((nC, nO, 1.0), (nO, N - nR, -1.0)):
        x = w - e[None, lo:hi] + sgn * Om[:, None]
        r2 = 2.0 * rho[:, p, lo:hi] ** 2
        if srg:
            f = 1.0 - torch.exp(-1000.0 * x * x)
            sig = sig + (r2 * f / x).sum()
            dsig = dsig - (r2 * f / (x * x)).sum()
        else:
            q = x * x + eta * eta
            sig = sig + (r2 * x / q).sum()
            dsig = dsig - (r2 * (x * x - eta * eta) / (q * q)).sum()
    return sig, dsig


def _x_self_energy(e, Om, rho, nC, nO, nR, eta, srg):
    N = e.numel()
    Sig = torch.zeros(N, dtype=F64, device=DEV)
    dS = torch.zeros(N, dtype=F64, device=DEV)
    for p in range(nC, N - nR):
        Sig[p], dS[p] = _x_poles(e, e[p], Om, rho, nC, nO, nR, p, eta, srg)
    x = e[None, nO:N - nR, None] - e[None, None, nC:nO] + Om[:, None, None]
    r2 = 4.0 * rho[:, nO:N - nR, nC:nO] ** 2
    f = (1.0 - torch.exp(-1000.0 * x * x)) / x if srg else x / (x * x + eta * eta)
    return Sig, 1.0 / (1.0 - dS), -float((r2 * f).sum())


def _x_newton(eHF, eW, Om, rho, nC, nO, nR, eta, srg, start, Z):
    eGW, Z = start.clone(), Z.clone()
    for p in range(nC, eHF.numel() - nR):
        w, f, n, df = float(start[p]), 1.0, 0, 1.0
        while abs(f) > 1e-6 and n < 64:
            n += 1
            sig, ds = _x_poles(eW, w, Om, rho, nC, nO, nR, p, eta, srg)
            both = torch.stack([sig, ds]).tolist()
            f = w - float(eHF[p]) - both[0]
            df = 1.0 / (1.0 - both[1])
            w -= df * f
        if n < 64:
            eGW[p], Z[p] = w, df
    return eGW, Z


def _x_ecrpa(L, e, nC, nO, nR):
    N = e.numel()
    if float(e[nO:N - nR].min()) <= float(e[nC:nO].max()):
        return float("nan")
    Om, _, trA, _ = _x_screening(L, e, nC, nO, nR)
    return 0.5 * (float(Om.sum()) - trA)


def _x_g0w0(c, L, e):
    nC, nO, nR = c.get("nC", 0), c["nO"], c.get("nR", 0)
    srg, eta = bool(c.get("reg", False)), c["eta"]
    Om, X, _, Lov = _x_screening(L, e, nC, nO, nR)
    rho = _x_rho(L, Lov, X)
    Sig, Z, gm = _x_self_energy(e, Om, rho, nC, nO, nR, eta, srg)
    if c.get("mixed"):
        # with eta = 0 the Newton search is a chaotic map for some orbitals: no such value
        return [None, None, None, Om, None, gm]
    lin = e + Z * Sig
    eGW, Zq = lin, Z
    if not c.get("linearize"):
        eGW, Zq = _x_newton(e, e, Om, rho, nC, nO, nR, eta, srg, lin, Z)
    return [eGW, Sig, Zq, Om, _x_ecrpa(L, eGW, nC, nO, nR), gm]


def _x_bse(c, L, e):
    nC, nO, nR, eta = c["nC"], c["nO"], c["nR"], c["eta"]
    N = c["N"]
    no, nv = nO - nC, N - nO - nR
    nS = no * nv
    Om, X, _, Lov = _x_screening(L, e, nC, nO, nR)
    rho = _x_rho(L, Lov, X)
    f = 4.0 * Om / (Om * Om + eta * eta)
    o, v = slice(nC, nO), slice(nO, N - nR)
    KA = torch.einsum("kij,kab->iajb", rho[:, o, o] * f[:, None, None], rho[:, v, v]).reshape(nS, nS)
    KB = torch.einsum("kib,kaj->iajb", rho[:, o, v] * f[:, None, None], rho[:, v, o]).reshape(nS, nS)
    K = Lov.T @ Lov                                                              # (ia|jb)
    Koovv = torch.einsum("Pij,Pab->iajb", L[:, o, o], L[:, v, v]).reshape(nS, nS)  # (ij|ab)
    Kx = K.reshape(no, nv, no, nv).permute(0, 3, 2, 1).reshape(nS, nS)             # (ib|ja)
    eG = torch.cat([e[:nO] - 0.05, e[nO:] + 0.05])
    d = (eG[None, v] - eG[o, None]).reshape(-1)
    out, ec = [], []
    for direct, mult in ((2.0, 1.0), (0.0, 3.0)):
        A = direct * K - Koovv + KA
        A.diagonal().add_(d)
        B = direct * K - Kx + KB
        C = torch.linalg.cholesky(A - B)
        w = torch.linalg.eigvalsh(C.T @ (A + B) @ C)
        Omx = w.sqrt()
        out.append(Omx)
        ec.append(mult * 0.5 * float(Omx.sum() - A.diagonal().sum()))
    return out + ec


def _x_evgw(c, L, e):
    nC, nO, nR, eta = c["nC"], c["nO"], c["nR"], c["eta"]
    eGW, n, conv = e.clone(), 0, 1.0
    while conv > 1e-5 and n <= c["maxSCF"]:
        Om, X, trA, Lov = _x_screening(L, eGW, nC, nO, nR)
        rho = _x_rho(L, Lov, X)
        Sig, Z, gm = _x_self_energy(eGW, Om, rho, nC, nO, nR, eta, False)
        new, Z = _x_newton(e, eGW, Om, rho, nC, nO, nR, eta, False, eGW, Z)
        conv = float((new - eGW).abs().max())
        eGW = new
        n += 1
    return [eGW, Sig, Z, 0.5 * (float(Om.sum()) - trA), gm, n]


def _x_qsgw(c, h):
    t = {k: torch.from_numpy(np.ascontiguousarray(h[k])).to(DEV) for k in
         ("eHF", "cHF", "PHF", "S", "T", "V", "Hc", "X", "ERI_AO")}
    S, E, X, nO, n, eta = t["S"], t["ERI_AO"], t["X"], h["nO"], h["nBas"], c["eta"]
    P, e, C, nSCF, conv = t["PHF"], t["eHF"], t["cHF"], -1, 1.0
    while conv > 1e-5 and nSCF < c["maxSCF"]:
        nSCF += 1
        J = torch.einsum("ls,mlns->mn", P, E)
        K = -torch.einsum("ls,mlsn->mn", P, E)
        M = E
        for _ in range(4):
            M = torch.tensordot(M, C, dims=([0], [0]))
        d = (e[None, nO:] - e[:nO, None]).reshape(-1)
        Kov = M[:nO, :nO, nO:, nO:].permute(0, 2, 1, 3).reshape(d.numel(), -1)   # (ia|jb) = <ij|ab>
        sq = d.sqrt()
        A2 = 4.0 * Kov * sq[:, None] * sq[None, :]
        A2.diagonal().add_(d * d)
        w, Zv = torch.linalg.eigh(A2)
        Om = w.abs().sqrt()
        XpY = Zv.T * sq[None, :] / Om.sqrt()[:, None]
        rho = torch.einsum("pjqb,mjb->mpq", M[:, :nO, :, nO:], XpY.reshape(-1, nO, n - nO))
        _, Z, gm = _x_self_energy(e, Om, rho, 0, nO, 0, eta, False)
        Sig = torch.zeros(n, n, dtype=F64, device=DEV)
        for lo, hi, sgn in ((0, nO, 1.0), (nO, n, -1.0)):
            x = e[None, :, None] - e[None, None, lo:hi] + sgn * Om[:, None, None]
            r = rho[:, :, lo:hi]
            Sig += 2.0 * torch.einsum("mpx,mqx->pq", r * x / (x * x + eta * eta), r)
        SC = S @ C
        SigP = SC @ (0.5 * (Sig + Sig.T)) @ SC.T
        F = t["Hc"] + J + 0.5 * K + SigP
        err = F @ P @ S - S @ P @ F
        if nSCF > 1:
            conv = float(err.abs().max())
        En = float((P * t["T"]).sum() + (P * t["V"]).sum() + 0.5 * (P * J).sum()
                   + 0.25 * (P * K).sum())
        ec = 0.5 * float(Om.sum() - (d + 2.0 * Kov.diagonal()).sum())
        e, cp = torch.linalg.eigh(X.T @ F @ X)
        C = X @ cp
        P = 2.0 * C[:, :nO] @ C[:, :nO].T
    return [e, P.reshape(-1), Z, En, ec, gm, nSCF]


def exact(case, seed):
    c = dict(case)
    kind = c["kind"]
    if kind in ("host", "g0w0", "g0w0_L"):
        return _x_g0w0(c, *_system(c, seed))
    if kind == "evgw_L":
        return _x_evgw(c, *_system(c, seed))
    if kind == "bse":
        return _x_bse(c, *_system(c, seed))
    if kind == "batch":
        got = [_x_g0w0(dict(c, nO=nO), L, e) for _, nO, L, e in _batch_systems(c, seed)]
        return [torch.cat([r[0] for r in got]), np.array([r[4] for r in got]),
                np.zeros(len(got), dtype=np.int64)]
    if kind == "qsgw":
        return _x_qsgw(c, _chain(c, seed))
    if kind == "aomo":
        coef, M = _aomo_inputs(c, seed)
        M = M.reshape((c["nBas"],) * 4)             # [s, r, q, p] of the Fortran tensor
        for _ in range(4):
            M = torch.tensordot(M, coef, dims=([0], [1]))
        return [M.reshape(-1)]
    e, Om, rho = _sigma_inputs(c, seed)
    rho = rho.transpose(1, 2)                       # rho[m, p, q] of the Fortran rho(p, q, m)
    Sig, Z, gm = _x_self_energy(e, Om, rho, 0, c["nO"], 0, c["eta"], False)
    return [torch.tensor([gm], dtype=F64), Sig, Z, 0]
