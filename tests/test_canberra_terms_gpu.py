"""Canberra's division route against its shared reciprocals."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


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
