"""The sums behind a variable's statistics: the norm to far better than r's own rounding,
and means far above the spread over millions of observations, against FP64."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [32, 64])
@pytest.mark.parametrize("offset", [0, 1])  # floats off a 16-byte boundary
def test_norms_do_not_bias_r(gpu, n, offset):
    """Whole numbers and a power of two of them: means and centred values are exact, their
    squares are not.  The rounding of r (2^-24 relative, uniform at most) averages
    to 2^-24 / sqrt(3 p) = 2^-30.3 over a variable's entries; what is left above that is
    the error of its norm."""
    import torch
    import gputools_gb300 as g
    p = 2048
    gen = torch.Generator(device="cuda").manual_seed(n + offset)
    whole = lambda *s: torch.randint(0, 4096, s, generator=gen, device="cuda").float()
    X = torch.empty(p * n + offset, device="cuda")[offset:].view(p, n)
    X.copy_(whole(1, n) + whole(p, n))
    old = g.get_gram_path()
    g.set_gram_path("f16x6")
    try:
        got = g.pmcc_device(X, outputs=("corr",))["corr"].double()
    finally:
        g.set_gram_path(old)
    Z = X.double()
    Z = Z - Z.mean(1, keepdim=True)
    Z = Z / Z.norm(dim=1, keepdim=True)
    want = Z @ Z.T
    use = (want.abs() >= 0.1).fill_diagonal_(False)
    rel = torch.where(use, got / want - 1.0, torch.zeros_like(want))
    bias = rel.sum(1) / use.sum(1)
    assert float(bias.square().mean().sqrt()) <= 2.0 ** -29


def test_mean_far_above_the_spread_of_many_observations(gpu):
    """4e6 +- 1 in steps of a float (0.5), 16 million times: the plain sum of the values
    is off by many spreads.  The gradient of the correlations scales with 1 / norm
    and its contraction runs over the four variables alone: operands of 2^-22, a few
    float roundings each of z, W and the result."""
    import torch
    p, n = 4, 16_000_000
    gen = torch.Generator(device="cuda").manual_seed(5)
    X = torch.randn((p, n), generator=gen, device="cuda")
    X[1:] += 0.7 * X[0]
    X += 4e6
    G = torch.randn((p, p), generator=gen, device="cuda")
    out = torch.empty_like(X)
    vp = lambda t: ctypes.c_void_p(t.data_ptr())
    st = gpu.gt_cor_backward_device(vp(X), p, n, vp(G), vp(out),
                                    ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert st == 0, gpu.gt_last_error().decode()
    C = X.double()
    C = C - C.mean(1, keepdim=True)
    s = C.norm(dim=1, keepdim=True)
    C = C / s
    W = (G + G.T).double() @ C
    want = (W - C * (C * W).sum(1, keepdim=True)) / s
    err = (out.double() - want).abs().amax(1) / want.abs().amax(1)
    assert float(err.max()) <= 4e-6


@pytest.mark.parametrize("log2scale", [118, 123, -115, -120])
def test_norms_near_the_ends_of_the_float_range(gpu, rng, log2scale):
    """1 / norm subnormal, or its low half: the error-free Gram's tolerance all the same."""
    import torch
    import gputools_gb300 as g
    p, n = 24, 1024
    X = (rng.standard_normal((1, n)) + rng.standard_normal((p, n))).astype(np.float32)
    Z = X.astype(np.float64)
    Z -= Z.mean(1, keepdims=True)
    Z /= np.linalg.norm(Z, axis=1, keepdims=True)
    want = Z @ Z.T
    np.fill_diagonal(want, 1.0)
    dX = torch.from_numpy(X * np.float32(2.0 ** log2scale)).cuda()
    old = g.get_gram_path()
    g.set_gram_path("f16x6")
    try:
        got = g.pmcc_device(dX, outputs=("corr",))["corr"].cpu().numpy()
    finally:
        g.set_gram_path(old)
    assert np.max(np.abs(got - want)) <= 1.5e-7


@pytest.mark.parametrize("path", ["f16x3", "fp32", "f16x6"])
@pytest.mark.parametrize("p,n", [(24, 64), (300, 40)])
def test_subnormal_values(gpu, rng, path, p, n):
    """Whole multiples of the smallest float: exact inputs of which 1 / norm overflows."""
    import torch
    import gputools_gb300 as g
    K = (rng.integers(-500, 500, (1, n)) + rng.integers(-500, 500, (p, n))).astype(np.float64)
    X = (K * 2.0 ** -149).astype(np.float32)
    Z = K - K.mean(1, keepdims=True)
    Z /= np.linalg.norm(Z, axis=1, keepdims=True)
    want = Z @ Z.T
    np.fill_diagonal(want, 1.0)
    old = g.get_gram_path()
    g.set_gram_path(path)
    try:
        got = g.pmcc_device(torch.from_numpy(X).cuda(), outputs=("corr",))["corr"].cpu().numpy()
    finally:
        g.set_gram_path(old)
    assert np.max(np.abs(got - want)) <= (1.5e-7 if path == "f16x6" else 3e-6)
