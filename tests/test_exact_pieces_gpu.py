"""The error-free Pearson Gram with its observations in pieces (few tiles): both kinds
of problem, ragged blocks and last pieces, missing-value gate, and NaN variables, at
the whole Gram's tolerance."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture
def exact(gpu):
    import gputools_gb300 as g
    old = g.get_gram_path()
    g.set_gram_path("f16x6")
    yield g
    g.set_gram_path(old)


def data(p, n, seed):
    import torch
    gen = torch.Generator(device="cuda").manual_seed(seed)
    X = torch.randn((p, n), generator=gen, device="cuda").add_(5).exp_()
    return X + 1000 * torch.rand((p, 1), generator=gen, device="cuda")


def reference(X, Y=None):
    def unit(A):
        A = A.double()
        A = A - A.mean(1, keepdim=True)
        return A / A.norm(dim=1, keepdim=True)
    Z = unit(X)
    r = Z @ (Z if Y is None else unit(Y)).T
    return r.fill_diagonal_(1.0) if Y is None else r


@pytest.mark.parametrize("p,n", [(2, 1024), (33, 1025), (129, 4160), (257, 9000), (700, 1999),
                                 (1025, 2049), (1500, 1100)])
def test_symmetric(exact, p, n):
    import torch
    X = data(p, n, p)
    got = exact.pmcc_device(X)
    assert float((got["corr"].double() - reference(X)).abs().max()) <= 1.5e-7
    assert torch.equal(got["corr"], got["corr"].T) and torch.equal(got["ts"], got["ts"].T)
    assert bool((got["pairs"] == n).all())


@pytest.mark.parametrize("nA,nB,n", [(1, 1, 1030), (129, 2000, 1600), (3, 2500, 5000), (1025, 31, 3000)])
def test_two_sets(exact, nA, nB, n):
    A, B = data(nA, n, 1), data(nB, n, 2)
    got = exact.pmcc_device(A, B, outputs=("corr",))["corr"]
    assert float((got.double() - reference(A, B)).abs().max()) <= 1.5e-7


def test_nan_and_constant_variables(exact):
    X = data(200, 3000, 9)
    X[7, 11] = float("nan")
    X[20] = 4.0
    r = exact.pmcc_device(X, outputs=("corr",))["corr"]
    bad = [7, 20]
    assert bool(r[bad].isnan().all()) and bool(r[:, bad].isnan().all())
    keep = [i for i in range(200) if i not in bad]
    got = r[keep][:, keep]
    assert float((got.double() - reference(X[keep])).abs().max()) <= 1.5e-7


def test_gated_by_the_missing_value_flag(exact):
    X = data(300, 2500, 5)
    got = exact.pmcc_device(X, use=1, outputs=("corr",))["corr"]
    assert float((got.double() - reference(X)).abs().max()) <= 1.5e-7
