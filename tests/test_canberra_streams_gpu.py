"""Canberra keeps nothing in the library's workspace, so that calls on different streams
are independent; the counts of its zeros from 512 coordinates on come from the points."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_no_device_memory_and_one_launch(gpu):
    import torch
    import gputools_gb300 as g
    P = torch.randn(500, 70, device="cuda").abs()
    out = torch.empty(500 * 500, device="cuda")
    g.distances_device(P, "canberra", layout="full", out=out)
    gpu.gt_release_workspace()
    torch.cuda.synchronize()
    free, launches = torch.cuda.mem_get_info()[0], gpu.gt_kernel_launches()
    g.distances_device(P, "canberra", layout="full", out=out)
    torch.cuda.synchronize()
    assert torch.cuda.mem_get_info()[0] == free
    assert gpu.gt_kernel_launches() == launches + 1


@pytest.mark.parametrize("n,d", [(70, 31), (65, 48), (66, 511), (130, 512), (64, 513), (67, 1030), (65, 1537)])
@pytest.mark.parametrize("scale", [1.0, 2.0 ** -40])  # shared reciprocals and divisions
def test_counts_of_zeros(gpu, oracle_mod, rng, n, d, scale):
    import torch
    import gputools_gb300 as g
    P = np.exp(rng.standard_normal((n, d))).astype(np.float32) * np.float32(scale)
    P[rng.random((n, d)) < 0.7] = 0
    P[1, 16:] = P[2, :-3] = 0
    P[5] = P[6] = 0
    want = oracle_mod.dist(P, "canberra")
    got = g.distances_device(torch.from_numpy(P).cuda(), "canberra",
                             layout="full").cpu().numpy().reshape(n, n).astype(np.float64)
    off = ~np.eye(n, dtype=bool)
    assert np.array_equal(np.isnan(got[off]), np.isnan(want[off])) and np.isnan(want[5, 6])
    ok = off & ~np.isnan(want)
    # a miscounted zero changes an entry by one part in d at least
    assert np.all(np.abs(got - want)[ok] <= (d + 8) * 2.0 ** -24 * want[ok])
