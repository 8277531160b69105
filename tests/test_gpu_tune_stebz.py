"""The tuned width of the FP64 bisection is relative to the best one of each size, so that a tuned
context and tables saved for an earlier kernel are no slower than an untuned one.
"""
import json

import numpy as np
import pytest

from quack_gb300 import api

pytestmark = pytest.mark.gpu


def _w(c, A):
    import torch
    n = A.shape[0]
    dA = torch.from_numpy(A.copy()).cuda()
    w = torch.empty(n, dtype=torch.float64, device="cuda")
    api.dsyev_dev(n, dA.data_ptr(), n, w.data_ptr(), 0, False, ctx=c)
    return w.cpu().numpy()


@pytest.mark.parametrize("n", [60, 600, 1300, 2000])
def test_relative_width(n):
    rng = np.random.default_rng(n)
    A = rng.standard_normal((n, n))
    A += A.T
    c = api.Context(0)
    try:
        dflt = c.tune_query("stebz_lanes", n)
        ref = _w(c, A)
        assert dflt in (8, 16, 32)
        for v, lanes in ((4, dflt), (2, dflt // 2), (8, min(32, 2 * dflt)), (1, max(4, dflt // 4)),
                         (32, 32)):
            c.tune_set("stebz_k", n, v)
            assert c.tune_query("stebz_lanes", n) == lanes
            # a bracket's middle is within 2^-52 of where the count changes, and that within 10 2^-53
            # ||T|| of the eigenvalue (three roundings a step of the recurrence), on both sides
            assert np.max(np.abs(_w(c, A) - ref)) <= 24 * 2.0 ** -53 * np.max(np.abs(ref))
    finally:
        c.close()


def test_tables(tmp_path):
    n = 600
    c = api.Context(0)
    try:
        dflt = c.tune_query("stebz_lanes", n)
        assert dflt >= 8
        old = tmp_path / "v1.json"
        old.write_text(json.dumps({"version": 1, "entries": [
            {"param": "sytrd_grid", "bucket": 9, "value": 3}, {"param": "stebz_k", "bucket": 9, "value": 2}]}))
        c.tune_load(old)
        assert c.tune_query("sytrd_grid", n) == 3
        assert c.tune_query("stebz_lanes", n) == dflt
        c.tune_set("stebz_k", n, 2)
        c.tune_save(tmp_path / "v2.json")
        c.tune_set("stebz_k", n, 4)
        c.tune_load(tmp_path / "v2.json")
        assert c.tune_query("stebz_k", n) == 2 and c.tune_query("stebz_lanes", n) == dflt // 2
    finally:
        c.close()
