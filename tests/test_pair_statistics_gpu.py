"""Per-variable statistics finished in float pairs: r of variables whose mean
dwarfs their spread, of constant variables, of extreme scales and of more
observations than a float counts exactly, against FP64."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def corr(X, path):
    import torch
    import gputools_gb300 as g
    old = g.get_gram_path()
    g.set_gram_path(path)
    try:
        return g.pmcc_device(torch.from_numpy(X).cuda(), outputs=("corr",))["corr"].cpu().numpy()
    finally:
        g.set_gram_path(old)


@pytest.mark.parametrize("n", [2, 3, 41, 47, 1000, 4099])
@pytest.mark.parametrize("scale", [1.0, 2.0 ** 100, 2.0 ** -100])
def test_large_offsets_and_scales(gpu, rng, n, scale):
    """Means of up to 2^18 times the spread: the float inputs are exact, so
    FP64 is; the error-free Gram leaves its final rounding (2^-24) and the
    statistics' share, |mean| / spread times 2^-46 and less."""
    base = rng.standard_normal((1, n))
    X = base + 0.5 * rng.standard_normal((20, n)) + 2.0 ** rng.integers(0, 19, (20, 1))
    X = (X * scale).astype(np.float32)
    got = corr(X, "f16x6")
    Z = X.astype(np.float64) / scale
    Z -= Z.mean(1, keepdims=True)
    Z /= np.linalg.norm(Z, axis=1, keepdims=True)
    want = Z @ Z.T
    np.fill_diagonal(want, 1.0)
    assert np.max(np.abs(got - want)) <= 1.5e-7


@pytest.mark.parametrize("n", [2, 41, 55, 61, 997, 8191])
def test_constant_variables_are_flagged(gpu, rng, n):
    X = rng.standard_normal((12, n)).astype(np.float32)
    X[::2] = rng.standard_normal((6, 1)).astype(np.float32) * np.float32(1e3)
    got = corr(X, "f16x3")
    assert np.all(np.isnan(got[::2])) and np.all(np.isnan(got[:, ::2]))
    assert np.all(np.isfinite(got[1::2, 1::2]))


def test_more_observations_than_a_float_counts(gpu):
    import torch
    import gputools_gb300 as g
    n = (1 << 24) + 3
    gen = torch.Generator(device="cuda").manual_seed(1)
    X = torch.randn((3, n), generator=gen, device="cuda") + 5.0
    X[1] += 0.3 * X[0]
    got = g.pmcc_device(X, outputs=("corr",))["corr"].double()
    want = torch.corrcoef(X.double())
    assert float((got - want).abs().max()) <= 1e-3  # f16x3 sums 2^24 products in float
