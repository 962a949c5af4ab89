"""Pairwise-complete Pearson at the edges of its tiles, stores and clusters: column
counts around 32 and 64, rows around 128, outputs with odd row strides, problems
below and above a cluster per pair of SMs, and its bounded waits, against float64."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GT_OK, GT_ETIMEOUT = 0, 5


def data(p, n, seed):
    import torch
    gen = torch.Generator(device="cuda").manual_seed(seed)
    X = torch.randn((p, n), generator=gen, device="cuda") * 2 + 5
    X[torch.rand((p, n), generator=gen, device="cuda") < 0.05] = float("nan")
    return X


def reference(X, Y):
    m, w = (~X.isnan()).double(), (~Y.isnan()).double()
    mu, nu = X.nanmean(1, keepdim=True), Y.nanmean(1, keepdim=True)
    x, y = (X - mu).nan_to_num(0).double(), (Y - nu).nan_to_num(0).double()
    N = m @ w.T
    sx, sy = x @ w.T, m @ y.T
    c = x @ y.T - sx * sy / N
    return c / ((x * x @ w.T - sx * sx / N) * (m @ (y * y).T - sy * sy / N)).sqrt(), N


def tol(n):  # the masked Gram carries the f16x3 split
    return 2e-6 * np.sqrt(max(n, 100) / 100.0) + 1e-6


@pytest.mark.parametrize("p,n", [(31, 80), (300, 257), (1024, 100), (1057, 64), (1200, 300), (1281, 70)])
def test_symmetric(gpu, p, n):
    import torch
    import gputools_gb300 as g
    X = data(p, n, p)
    got = g.pmcc_device(X, use=1)
    r, N = reference(X, X)
    assert torch.equal(got["pairs"].double(), N)
    assert float((got["corr"].double() - r.clamp(-1, 1)).abs().max()) <= tol(n)
    for k in ("corr", "pairs"):
        assert torch.equal(got[k], got[k].T)


@pytest.mark.parametrize("nA,nB,n", [(129, 2500, 90), (3, 6000, 64), (513, 1056, 129), (100, 200, 300)])
def test_two_sets(gpu, nA, nB, n):
    import torch
    import gputools_gb300 as g
    A, B = data(nA, n, 1), data(nB, n, 2)
    got = g.pmcc_device(A, B, use=1)
    r, N = reference(A, B)
    assert torch.equal(got["pairs"].double(), N)
    assert float((got["corr"].double() - r.clamp(-1, 1)).abs().max()) <= tol(n)


def test_short_wait_limit_reports_timeout_and_recovers(gpu):
    import torch
    import gputools_gb300 as g
    X = data(2000, 2000, 3)
    lib = g.load()
    sp = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    assert lib.gt_device_status(sp) == GT_OK
    seen = set()
    try:
        assert lib.gt_set_wait_limit_ns(2000) == GT_OK
        for _ in range(3):
            g.pmcc_device(X, use=1, outputs=("corr",))
            seen.add(lib.gt_device_status(sp))
    finally:
        lib.gt_set_wait_limit_ns(0)
    assert seen <= {GT_OK, GT_ETIMEOUT} and GT_ETIMEOUT in seen
    got = g.pmcc_device(X, use=1, outputs=("corr",))["corr"]
    assert lib.gt_device_status(sp) == GT_OK
    assert float((got.double() - reference(X, X)[0].clamp(-1, 1)).abs().max()) <= tol(2000)
