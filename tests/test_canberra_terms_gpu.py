"""Canberra of few coordinates: every term a subtraction, an addition and a division, the
sum d - 1 additions more, each rounded once (2^-24 relative of a sum of positive
terms)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d", [1, 2, 3, 7])
@pytest.mark.parametrize("layout", ["full", "dist"])
def test_roundings_of_few_coordinates(gpu, rng, d, layout):
    import torch
    import gputools_gb300 as g
    n = 700
    P = np.exp(rng.standard_normal((n, d))).astype(np.float32)
    got = g.distances_device(torch.from_numpy(P).cuda(), "canberra", layout=layout).cpu().numpy()
    A = P.astype(np.float64)
    want = sum(np.abs(A[:, None, k] - A[None, :, k]) / (A[:, None, k] + A[None, :, k])
               for k in range(d))
    i, j = np.triu_indices(n, 1)
    got = got.reshape(n, n)[i, j] if layout == "full" else got
    want = want[i, j]
    assert np.all(np.abs(got - want) <= (d + 2) * 1.0001 * 2.0 ** -24 * want)


@pytest.mark.parametrize("scale", [2.0 ** -40, 2.0 ** 70])
@pytest.mark.parametrize("n,d", [(65, 8), (130, 17), (64, 48), (200, 33)])
def test_scale_does_not_matter(gpu, rng, scale, n, d):
    """Values all outside the shared reciprocal's range: the divisions, zeros among them,
    give the distances of the same values within it (each within d + 8 roundings)."""
    import torch
    import gputools_gb300 as g
    P = rng.standard_normal((n, d)).astype(np.float32)
    P[rng.random((n, d)) < 0.3] = 0
    P[3] = P[0] = 0
    run = lambda X: g.distances_device(torch.from_numpy(X).cuda(), "canberra",
                                       layout="full").cpu().numpy().astype(np.float64)
    a, b = run(P), run((P * np.float32(scale)).astype(np.float32))
    assert np.array_equal(np.isnan(a), np.isnan(b)) and np.isnan(a).any()
    ok = np.isfinite(a)
    assert np.all(np.abs(a - b)[ok] <= 2 * (d + 8) * 2.0 ** -24 * a[ok])
