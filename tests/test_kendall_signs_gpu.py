"""Kendall's counts as an FP8 Gram of pair signs: bit-exact tau-b at the edges
of the 128 x 256 tiles, of the four-byte sign groups and of the row segments,
and where the sums are largest."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def device_tau(X, Y=None):
    import torch
    import gputools_gb300 as g
    dX = torch.from_numpy(X).cuda()
    dY = None if Y is None else torch.from_numpy(Y).cuda()
    return g.kendall_device(dX, dY).cpu().numpy()


def same_bits(a, b):
    return np.array_equal(a, b, equal_nan=True)


@pytest.mark.parametrize("p,n", [(1, 2), (127, 6), (128, 7), (129, 9), (256, 65), (257, 130),
                                 (385, 33), (3, 1023), (3, 1025), (2, 2051)])
def test_tile_and_segment_edges(gpu, oracle_mod, rng, p, n):
    X = rng.integers(0, 6, (p, n)).astype(np.float32)
    want, *_ = oracle_mod.kendall(X)
    assert same_bits(device_tau(X), want)


@pytest.mark.parametrize("nx,ny,n", [(1, 300, 21), (300, 1, 22), (130, 129, 500), (5, 260, 1030)])
def test_two_sets(gpu, oracle_mod, rng, nx, ny, n):
    X = rng.standard_normal((nx, n)).astype(np.float32)
    Y = rng.integers(0, 3, (ny, n)).astype(np.float32)
    want, *_ = oracle_mod.kendall(X, Y)
    assert same_bits(device_tau(X, Y), want)


def test_infinities_and_signed_zeros(gpu, oracle_mod, rng):
    X = rng.choice(np.array([-np.inf, -1e-45, -0.0, 0.0, 1e-45, 2.0, np.inf], np.float32), (9, 101))
    want, *_ = oracle_mod.kendall(X)
    assert same_bits(device_tau(X), want)


@pytest.mark.parametrize("p,n", [(40, 6000), (6200, 700)])
def test_largest_sums_are_exact(gpu, p, n):
    """Increasing and decreasing variables: every |S| is n (n - 1) / 2, the
    largest possible, in one piece of K (6200 variables) and in many."""
    sign = np.where(np.random.default_rng(p).random(p) < 0.5, -1.0, 1.0)
    X = np.ascontiguousarray((sign[:, None] * np.arange(n)[None]).astype(np.float32))
    total = n * (n - 1) / 2
    v = min(1.0, total / (np.sqrt(total) * np.sqrt(total)))
    want = sign[:, None] * sign[None] * v
    np.fill_diagonal(want, 1.0)
    assert same_bits(device_tau(X), want)
