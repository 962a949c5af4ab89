"""f16x3 Pearson on either side of its dispatch limits: which kernels ran, from their
launches or from bits that only one of them gives, and r on both sides against FP64."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def values(p, n, seed=1):
    import torch
    gen = torch.Generator(device="cuda").manual_seed(seed)
    X = torch.randn((p, n), generator=gen, device="cuda")
    return X + 0.8 * torch.randn((1, n), generator=gen, device="cuda") + 3.0


def corr(A, B=None):
    """r, checked against FP64 (at most 400 rows), and the launches it took."""
    import torch
    import gputools_gb300 as g
    lib = g.load()
    assert g.get_gram_path() == "f16x3"
    before = lib.gt_kernel_launches()
    got = g.pmcc_device(A, B, outputs=("corr",))["corr"]
    launches = lib.gt_kernel_launches() - before
    unit = lambda X: torch.nn.functional.normalize(X.double() - X.double().mean(1, keepdim=True))
    rows = torch.arange(0, A.shape[0], max(1, A.shape[0] // 400), device="cuda")
    want = unit(A)[rows] @ unit(A if B is None else B).T
    tol = 2e-6 * np.sqrt(max(A.shape[1], 100) / 100.0) + 1e-6
    assert float((got[rows].double() - want).abs().max()) <= tol
    return got, launches


@pytest.mark.parametrize("p,n", [(1000, 240),   # 2.4e8 products
                                 (1581, 90)])   # 2.5e6 entries
def test_products_and_entries_of_the_multiply_adds(gpu, p, n):
    """The entries of the first p - 1 variables are the same bits among p - 1 and p (both
    FP32 multiply-adds) and among p + 1 and p + 2 (both tensor cores), not across."""
    import torch
    X = values(p + 2, n)
    r = {q: corr(X[:q].contiguous())[0][:p - 1, :p - 1] for q in (p - 1, p, p + 1, p + 2)}
    assert torch.equal(r[p - 1], r[p])
    assert torch.equal(r[p + 1], r[p + 2])
    assert not torch.equal(r[p], r[p + 1])


def test_observations_of_the_multiply_adds(gpu):
    # statistics and products; on the tensor cores the pieces are added by a third
    assert [corr(values(100, n))[1] for n in (1500, 1501)] == [2, 3]
    # both sets' statistics in one launch; two prologues there
    two = lambda n: corr(values(50, n), values(60, n, seed=2))[1]
    assert [two(n) for n in (2000, 2001)] == [2, 4]


@pytest.mark.parametrize("p,q,n", [
    (2560, 0, 1024),     # 55 pairs of tiles: single CTAs
    (2561, 0, 1024),     # 66, four fifths of 76: pairs of CTAs from 1024 observations
    (2700, 0, 960), (2700, 0, 1000), (2700, 0, 2047),
    (2816, 0, 1025), (2817, 0, 300),   # 78: pairs at any length
    (2048, 1900, 1024),  # 64 of two sets
])
def test_pairs_of_ctas_for_four_fifths_of_the_chip(gpu, p, q, n):
    corr(values(p, n), values(q, n, seed=2) if q else None)
