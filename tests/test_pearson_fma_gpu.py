"""Small "everything" Pearson problems as FP32 multiply-adds: edges of the 32 x 32
tiles and of the slabs of 32 observations, both kinds of problem, outputs left
out, and both sides of the limit to the tensor-core Gram."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# z and its products are rounded to 2^-24 each, sums of 32 and their sums add at
# most (n / 128 + 32 + 8) * 2^-24 of sum |z_x z_y| <= 1
def tol(n):
    return (n / 128 + 48) * 2.0 ** -24


def expression(rng, p, n):
    return (np.exp(rng.standard_normal((p, n))) * 100 + rng.uniform(0, 1000, (p, 1))).astype(np.float32)


def check(got, want, n):
    assert np.array_equal(np.isnan(got["corr"]), np.isnan(want))
    ok = ~np.isnan(want)
    r = got["corr"][ok]
    assert np.abs(r - want[ok]).max() <= tol(n)
    assert np.all(got["pairs"] == n)
    t = got["ts"][ok]
    far = np.abs(r) < 0.99
    rule = r[far].astype(np.float64) * np.sqrt((n - 2) / (1 - r[far].astype(np.float64) ** 2))
    assert np.allclose(t[far], rule, rtol=2e-6, atol=1e-6)
    assert np.all(t[r >= 0.999] == 10000)


def run(X, Y=None):
    import torch
    import gputools_gb300 as g
    dX = torch.from_numpy(X).cuda()
    dY = None if Y is None else torch.from_numpy(Y).cuda()
    return {k: v.cpu().numpy() for k, v in g.pmcc_device(dX, dY).items()}


@pytest.mark.parametrize("p", [1, 31, 32, 33, 65, 130])
@pytest.mark.parametrize("n", [3, 31, 32, 33, 96, 129, 1001])
def test_symmetric(gpu, oracle_mod, rng, p, n):
    X = expression(rng, p, n)
    if p > 40:
        X[3] = 7.0            # constant
        X[5, n // 2] = np.nan
    want, _, _ = oracle_mod.pearson(X)
    got = run(X)
    check(got, want, n)
    if p > 1:
        assert np.array_equal(got["corr"], got["corr"].T, equal_nan=True)
        assert np.all(np.diag(got["corr"])[~np.isnan(np.diag(want))] == 1.0)


@pytest.mark.parametrize("nA,nB,n", [(1, 1, 4), (33, 1, 40), (1, 95, 64), (64, 97, 200), (2500, 3, 37)])
def test_two_sets(gpu, oracle_mod, rng, nA, nB, n):
    X, Y = expression(rng, nA, n), expression(rng, nB, n)
    want, _, _ = oracle_mod.pearson(X, Y)
    check(run(X, Y), want, n)


@pytest.mark.parametrize("p,n", [(1000, 500), (1000, 501), (100, 4096), (100, 4097)])
def test_both_sides_of_the_limit(gpu, oracle_mod, rng, p, n):
    X = expression(rng, p, n)
    rows = np.array([0, 1, p // 2, p - 1])
    want, _, _ = oracle_mod.pearson(X[rows], X)
    got = run(X)["corr"][rows]
    want[np.arange(4), rows] = 1.0
    assert np.abs(got - want).max() <= 2e-6 * np.sqrt(n / 100.0) + 1e-6


def test_outputs_left_out(gpu, rng):
    import torch
    import gputools_gb300 as g
    X = torch.from_numpy(expression(rng, 50, 60)).cuda()
    full = g.pmcc_device(X)
    for k in full:
        assert torch.equal(g.pmcc_device(X, outputs=(k,))[k], full[k])
