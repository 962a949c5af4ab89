"""The error-free Gram on pairs of CTAs (256 x 256 tiles, cta_group::2): edges of
the row blocks, both kinds of problem, the smallest problems that take it, and
its bounded waits."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GT_OK, GT_ETIMEOUT = 0, 5


@pytest.fixture
def exact_path():
    import gputools_gb300 as g
    old = g.get_gram_path()
    g.set_gram_path("f16x6")
    yield g
    g.set_gram_path(old)


def reference(X, Y=None):
    def unit(A):
        A = A.double()
        A = A - A.mean(1, keepdim=True)
        return A / A.norm(dim=1, keepdim=True)
    Z = unit(X)
    r = Z @ (Z if Y is None else unit(Y)).T
    return r.fill_diagonal_(1.0) if Y is None else r


def data(p, n, seed):
    import torch
    gen = torch.Generator(device="cuda").manual_seed(seed)
    X = torch.randn((p, n), generator=gen, device="cuda").add_(5).exp_()
    return X + 1000 * torch.rand((p, 1), generator=gen, device="cuda")


@pytest.mark.parametrize("p,n", [(2817, 2), (2944, 64), (2945, 65), (3073, 127), (3200, 1000)])
def test_symmetric(gpu, exact_path, p, n):
    import torch
    X = data(p, n, p)
    got = exact_path.pmcc_device(X)
    assert float((got["corr"].double() - reference(X)).abs().max()) <= 1.5e-7
    assert torch.equal(got["corr"], got["corr"].T)
    assert bool((got["pairs"] == n).all())


@pytest.mark.parametrize("nA,nB,n", [(129, 19500, 40), (257, 10000, 96), (2500, 2100, 130)])
def test_two_sets(gpu, exact_path, nA, nB, n):
    A, B = data(nA, n, 1), data(nB, n, 2)
    got = exact_path.pmcc_device(A, B, outputs=("corr",))["corr"]
    assert float((got.double() - reference(A, B)).abs().max()) <= 1.5e-7


def test_short_wait_limit_reports_timeout_and_recovers(gpu, exact_path):
    import torch
    X = data(3000, 2048, 3)
    lib = exact_path.load()
    sp = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    assert lib.gt_device_status(sp) == GT_OK
    seen = set()
    try:
        assert lib.gt_set_wait_limit_ns(2000) == GT_OK
        for _ in range(3):
            exact_path.pmcc_device(X, outputs=("corr",))
            seen.add(lib.gt_device_status(sp))
    finally:
        lib.gt_set_wait_limit_ns(0)
    assert seen <= {GT_OK, GT_ETIMEOUT} and GT_ETIMEOUT in seen
    got = exact_path.pmcc_device(X, outputs=("corr",))["corr"]
    assert lib.gt_device_status(sp) == GT_OK
    assert float((got.double() - reference(X)).abs().max()) <= 1.5e-7
