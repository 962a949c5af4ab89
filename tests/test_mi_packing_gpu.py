"""gpuMi's operand packing: 32 / stride whole variables to a group of 32 rows.
Every row count (1, 2, 4, 5, 6, 8, 10, 16, 32) with full and partly filled last
groups, against the FP64 oracle, at gpuMi's tolerance."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bins,order", [(1, 1), (2, 2), (3, 1), (4, 3), (5, 2), (6, 4), (7, 3), (8, 8),
                                        (9, 3), (10, 1), (12, 5), (16, 2), (17, 3), (32, 6)])
@pytest.mark.parametrize("nx,ny,n", [(33, 0, 65), (1, 7, 20), (31, 130, 300)])
def test_packed_groups(gpu, oracle_mod, rng, bins, order, nx, ny, n):
    import torch
    import gputools_gb300 as g
    common = rng.standard_normal((1, n))
    X = (common + 0.5 * rng.standard_normal((nx, n))).astype(np.float32)
    Y = (common + 0.5 * rng.standard_normal((ny, n))).astype(np.float32) if ny else None
    want, _, _ = oracle_mod.bspline_mi(X, Y, bins=bins, order=order)
    got = g.mutual_info_device(torch.from_numpy(X).cuda(), None if Y is None else torch.from_numpy(Y).cuda(),
                               bins=bins, order=order).cpu().numpy().astype(np.float64)
    assert got.shape == want.shape
    assert np.all(np.abs(got - want) <= 3e-5 + 1e-4 * np.abs(want))
