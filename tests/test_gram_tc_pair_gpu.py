"""The split (f16x3, bf16x6, bf16x3) Grams on pairs of CTAs (256 x 256 tiles): edges of the
row blocks in both kinds of problem, the smallest problems that take it, short
and odd K, mutual information's operand, and its bounded waits."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GT_OK, GT_ETIMEOUT = 0, 5


@pytest.fixture
def lib_path():
    import gputools_gb300 as g
    old = g.get_gram_path()
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
    return torch.randn((p, n), generator=gen, device="cuda") + 3


def tol(path, n):  # the split Grams' tolerances, as for the single-CTA kernel
    return 2e-5 if path == "bf16x3" else 2e-6 * np.sqrt(n / 100.0) + 1e-6


@pytest.mark.parametrize("path", ["f16x3", "bf16x6", "bf16x3"])
@pytest.mark.parametrize("p,n", [(2817, 700), (2944, 2), (3073, 65), (3200, 1000)])
def test_symmetric(gpu, lib_path, path, p, n):
    import torch
    lib_path.set_gram_path(path)
    X = data(p, n, p)
    got = lib_path.pmcc_device(X)
    assert float((got["corr"].double() - reference(X)).abs().max()) <= tol(path, max(n, 100))
    assert torch.equal(got["corr"], got["corr"].T)
    assert bool((got["pairs"] == n).all())


@pytest.mark.parametrize("path", ["f16x3", "bf16x6", "bf16x3"])
@pytest.mark.parametrize("nA,nB,n", [(129, 19500, 400), (257, 10000, 96), (2500, 2100, 130)])
def test_two_sets(gpu, lib_path, path, nA, nB, n):
    lib_path.set_gram_path(path)
    A, B = data(nA, n, 1), data(nB, n, 2)
    got = lib_path.pmcc_device(A, B, outputs=("corr",))["corr"]
    assert float((got.double() - reference(A, B)).abs().max()) <= tol(path, max(n, 100))


@pytest.mark.parametrize("bins,order,nx,ny", [(10, 3, 700, 0), (16, 2, 500, 0), (4, 2, 1400, 0),
                                              (7, 3, 300, 900)])
def test_mutual_information(gpu, lib_path, bins, order, nx, ny):
    # 40 variables from all over a problem large enough for pairs, against the
    # same 40 in a problem of their own; gpuMi's tolerance
    import torch
    X = data(nx, 200, 5)
    Y = data(ny, 200, 6) if ny else None
    ix = torch.linspace(0, nx - 1, 40, device="cuda").long()
    iy = torch.linspace(0, ny - 1, 40, device="cuda").long() if ny else ix
    big = lib_path.mutual_info_device(X, Y, bins=bins, order=order)
    few = lib_path.mutual_info_device(X[ix].contiguous(), Y[iy].contiguous() if ny else None,
                                      bins=bins, order=order)
    sub = big[iy][:, ix] if big.shape[0] == (ny or nx) else big[ix][:, iy]
    assert sub.shape == few.shape
    assert bool(((sub - few).abs() <= 3e-5 + 1e-4 * few.abs()).all())


def test_short_wait_limit_reports_timeout_and_recovers(gpu, lib_path):
    import torch
    lib_path.set_gram_path("f16x3")
    X = data(3000, 2048, 3)
    lib = lib_path.load()
    sp = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    assert lib.gt_device_status(sp) == GT_OK
    seen = set()
    try:
        assert lib.gt_set_wait_limit_ns(2000) == GT_OK
        for _ in range(3):
            lib_path.pmcc_device(X, outputs=("corr",))
            seen.add(lib.gt_device_status(sp))
    finally:
        lib.gt_set_wait_limit_ns(0)
    assert seen <= {GT_OK, GT_ETIMEOUT} and GT_ETIMEOUT in seen
    got = lib_path.pmcc_device(X, outputs=("corr",))["corr"]
    assert lib.gt_device_status(sp) == GT_OK
    assert float((got.double() - reference(X)).abs().max()) <= tol("f16x3", 2048)
