"""Canberra's two routes, one reciprocal per two terms (slabs of 16 coordinates
whose values are zero or of magnitude 2^-30 to 2^60) and a division per term (any other
slab), against the oracle, alone and mixed within one sum."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def distances(P, layout="full"):
    import torch
    import gputools_gb300 as g
    return g.distances_device(torch.from_numpy(P).cuda(), "canberra", layout=layout).cpu().numpy()


def abundances(rng, n, d, zeros):
    x = np.exp(rng.standard_normal((n, d))).astype(np.float32)
    x[rng.random((n, d)) < zeros] = 0
    return x


def check(oracle_mod, P):
    """Each of d terms is within 5 roundings, the sum makes at most d more,
    the rescaling 2."""
    n, d = P.shape
    want = oracle_mod.dist(P, "canberra")
    got = distances(P).reshape(n, n).astype(np.float64)
    tol = (d + 8) * 2.0 ** -24
    off = ~np.eye(n, dtype=bool)
    assert np.array_equal(np.isnan(got[off]), np.isnan(want[off]))
    fine = off & np.isfinite(want)
    assert np.array_equal(got[off & np.isinf(want)], want[off & np.isinf(want)])
    assert np.all(np.abs(got[fine] - want[fine]) <= tol * want[fine])
    i, j = np.triu_indices(n, 1)
    assert np.array_equal(distances(P, "dist"), got[j, i].astype(np.float32), equal_nan=True)


@pytest.mark.parametrize("n,d", [(2, 1), (63, 2), (65, 15), (64, 16), (130, 17), (70, 33), (129, 64)])
@pytest.mark.parametrize("zeros", [0.0, 0.3, 0.95])
def test_abundances(gpu, oracle_mod, rng, n, d, zeros):
    check(oracle_mod, abundances(rng, n, d, zeros))


def test_edges_of_the_range(gpu, oracle_mod, rng):
    """The largest and smallest values that share a reciprocal, beside zeros."""
    P = rng.choice(np.array([0.0, 2.0 ** -30, 2.0 ** 60, 1.0], np.float32), (80, 48))
    check(oracle_mod, P)


@pytest.mark.parametrize("bad", [-1.0, 1e-30, 1e-44, 1e30, np.inf])
def test_slabs_of_both_routes(gpu, oracle_mod, rng, bad):
    """One coordinate of the second of three slabs is out of the range in some points."""
    P = abundances(rng, 90, 40, 0.2)
    P[::7, 20] = bad
    check(oracle_mod, P)


def test_signed_values(gpu, oracle_mod, rng):
    """Both signs, with opposite values (a zero denominator only: infinite)."""
    P = rng.integers(-3, 4, (70, 12)).astype(np.float32)
    check(oracle_mod, P)
