"""The cached evGW graph against calls that come between two of its replays: a call that grows the
workspace, another caller buffer, a changed setting.  The replay runs the kernels of the eager
cycles in the same order, so the results are the same bits.
"""
import numpy as np
import pytest

from quack_gb300 import api, synth

pytestmark = pytest.mark.gpu
N, NO, NAUX = 40, 5, 120


def _inputs():
    import torch
    s = synth.gen_system(N, NO, NAUX, np.random.default_rng(11))
    dL = torch.from_numpy(api.L_fortran_flat(s["L"] * 0.4)).cuda()
    return dL, torch.from_numpy(s["eHF"]).cuda()


def _evgw(c, opts, dL, de, out):
    for t in out:
        t.zero_()
    r = api.evRGW_L_dev(opts, N, 0, NO, 0, NAUX, dL.data_ptr(), de.data_ptr(),
                        *[t.data_ptr() for t in out], ctx=c, raise_on_fail=False)
    return [t.cpu().numpy() for t in out] + [r["EcRPA"], r["EcGM"], r["nSCF"]]


def _same(a, b):
    return all(np.array_equal(x, y) for x, y in zip(a, b))


def _aomo(c, n):
    import torch
    C = torch.eye(n, dtype=torch.float64, device="cuda")
    E = torch.ones(n ** 4, dtype=torch.float64, device="cuda")
    M = torch.empty_like(E)
    api.AOtoMO_ERI_RHF_dev(n, n, C.data_ptr(), E.data_ptr(), M.data_ptr(), ctx=c)


def _g0w0(c, n, nO, naux):
    import torch
    s = synth.gen_system(n, nO, naux, np.random.default_rng(5))
    dL = torch.from_numpy(api.L_fortran_flat(s["L"] * 0.4)).cuda()
    de = torch.from_numpy(s["eHF"]).cuda()
    out = [torch.empty(k, dtype=torch.float64, device="cuda") for k in (n, n, n, nO * (n - nO))]
    api.RG0W0_L_dev(api.GWOptions(eta=0.1, linearize=True), n, 0, nO, 0, naux, dL.data_ptr(),
                    de.data_ptr(), *[t.data_ptr() for t in out], ctx=c)


# the transformation grows the digit planes, the larger G0W0 all of the eigensolver's workspace
@pytest.mark.parametrize("between", [lambda c: _aomo(c, 64), lambda c: _g0w0(c, 72, 9, 100)])
@pytest.mark.parametrize("linearize", [True, False])
def test_workspace_growth_between_replays(between, linearize):
    import torch
    opts = api.GWOptions(eta=0.1, maxSCF=4, linearize=linearize)
    dL, de = _inputs()
    out = [torch.empty(N, dtype=torch.float64, device="cuda") for _ in range(3)]
    c = api.Context(0)
    try:
        ref = _evgw(c, opts, dL, de, out)
        c.set_graph_mode(True)
        assert _same(_evgw(c, opts, dL, de, out), ref)
        between(c)
        # what the context gave back may go to the caller: these must stay as they are
        mine = [torch.full((1 << 22,), 7.0, dtype=torch.float64, device="cuda") for _ in range(16)]
        assert _same(_evgw(c, opts, dL, de, out), ref)
        assert all(bool((t == 7.0).all()) for t in mine)
    finally:
        c.close()


def test_other_output_buffers_and_settings():
    import torch
    opts = api.GWOptions(eta=0.1, maxSCF=4)
    dL, de = _inputs()
    out = [torch.empty(N, dtype=torch.float64, device="cuda") for _ in range(3)]
    other = [out[0]] + [torch.empty_like(t) for t in out[1:]]
    c = api.Context(0)
    try:
        ref = _evgw(c, opts, dL, de, out)
        c.tune_set("newton_maxit", 0, 2)
        ref2 = _evgw(c, opts, dL, de, out)
        c.tune_set("newton_maxit", 0, 64)
        assert not _same(ref, ref2)
        c.set_graph_mode(True)
        assert _same(_evgw(c, opts, dL, de, out), ref)
        assert _same(_evgw(c, opts, dL, de, other), ref)
        c.tune_set("newton_maxit", 0, 2)
        assert _same(_evgw(c, opts, dL, de, out), ref2)
    finally:
        c.close()
