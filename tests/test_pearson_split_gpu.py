"""The f16x3 Pearson Gram with its observations cut into pieces (few tiles): both
kinds of problem, ragged blocks and last pieces, from two pieces to the most, with
outputs left out, gated by the missing-value flag, and its bounded waits."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GT_OK, GT_ETIMEOUT = 0, 5


def data(p, n, seed):
    import torch
    gen = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randn((p, n), generator=gen, device="cuda") + 3


def reference(X, Y=None):
    def unit(A):
        A = A.double()
        A = A - A.mean(1, keepdim=True)
        return A / A.norm(dim=1, keepdim=True)
    Z = unit(X)
    r = Z @ (Z if Y is None else unit(Y)).T
    return r.fill_diagonal_(1.0) if Y is None else r


def tol(n):  # the f16x3 Gram's
    return 2e-6 * np.sqrt(n / 100.0) + 1e-6


def check(got, ref, n, sym):
    import torch
    r = got["corr"].double()
    assert float((r - ref).abs().max()) <= tol(n)
    if sym:
        assert torch.equal(got["corr"], got["corr"].T) and torch.equal(got["ts"], got["ts"].T)
    assert bool((got["pairs"] == n).all())
    far = r.abs() < 0.999  # the t-score's own formula, with its approximate root
    want = r * ((n - 2) / (1 - r * r)).sqrt()
    err = (got["ts"].double() - want).abs() <= 1e-5 * want.abs() + 1e-30
    assert bool((err | ~far).all())


@pytest.mark.parametrize("p,n", [(2, 5000), (33, 4999), (129, 4160), (257, 20000), (725, 1000),
                                 (1000, 577), (1701, 321), (1500, 4100)])
def test_symmetric(gpu, p, n):
    import gputools_gb300 as g
    X = data(p, n, p)
    check(g.pmcc_device(X), reference(X), n, True)


@pytest.mark.parametrize("nA,nB,n", [(1, 1, 4200), (129, 3000, 700), (3, 2000, 6000), (1025, 31, 9000)])
def test_two_sets(gpu, nA, nB, n):
    import gputools_gb300 as g
    A, B = data(nA, n, 1), data(nB, n, 2)
    check(g.pmcc_device(A, B), reference(A, B), n, False)


@pytest.mark.parametrize("missing", [False, True])
def test_gated(gpu, missing):
    # pairwise.complete.obs: the pieces' kernels run without a missing value only
    import torch
    import gputools_gb300 as g
    X = data(300, 5000, 7)
    if missing:
        X[5, 100] = float("nan")
    got = g.pmcc_device(X, use=1, outputs=("corr",))["corr"]
    ref = reference(X.nan_to_num(0))
    keep = torch.ones(300, dtype=torch.bool, device="cuda")
    keep[5] = not missing
    assert float((got.double() - ref)[keep][:, keep].abs().max()) <= tol(5000)
    if missing:
        Y = X[:, torch.arange(5000, device="cuda") != 100]
        assert float((got[5].double() - reference(Y)[5])[keep].abs().max()) <= tol(5000)


def test_short_wait_limit_reports_timeout_and_recovers(gpu):
    import torch
    import gputools_gb300 as g
    X = data(700, 20000, 3)
    lib = g.load()
    sp = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    assert lib.gt_device_status(sp) == GT_OK
    seen = set()
    try:
        assert lib.gt_set_wait_limit_ns(1000) == GT_OK
        for _ in range(3):
            g.pmcc_device(X, outputs=("corr",))
            seen.add(lib.gt_device_status(sp))
    finally:
        lib.gt_set_wait_limit_ns(0)
    assert seen <= {GT_OK, GT_ETIMEOUT}
    got = g.pmcc_device(X, outputs=("corr",))["corr"]
    assert lib.gt_device_status(sp) == GT_OK
    assert float((got.double() - reference(X)).abs().max()) <= tol(20000)
