"""Waits that give up after the producer has issued its last copy: with few observations
every copy of a tile is in flight at once, and a 200 ns limit ends before the first
arrives.  The CTA must wait for them all the same; the next call is bit-identical to
the one before."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GT_OK, GT_ETIMEOUT = 0, 5


@pytest.mark.parametrize("path,use,p,n", [
    ("f16x3", 0, 1700, 60),   # one tile each, two k-blocks
    ("f16x3", 0, 1700, 300),  # in pieces of the observations
    ("bf16x6", 0, 300, 60),
    ("f16x6", 0, 300, 100),
    ("f16x3", 1, 300, 60),    # pairwise, with missing values
])
def test_copies_in_flight_are_waited_for(gpu, rng, path, use, p, n):
    import torch
    import gputools_gb300 as g
    X = rng.standard_normal((p, n)).astype(np.float32)
    if use:
        X[rng.random(X.shape) < 0.05] = np.nan
    X = torch.from_numpy(X).cuda()
    sp = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    old = g.get_gram_path()
    g.set_gram_path(path)
    try:
        before = g.pmcc_device(X, use=use)
        assert gpu.gt_device_status(sp) == GT_OK
        seen = set()
        try:
            assert gpu.gt_set_wait_limit_ns(200) == GT_OK
            for _ in range(3):
                g.pmcc_device(X, use=use)
                seen.add(gpu.gt_device_status(sp))
        finally:
            gpu.gt_set_wait_limit_ns(0)
        assert GT_ETIMEOUT in seen, "a 200 ns limit never gave up a wait"
        after = g.pmcc_device(X, use=use)
        assert gpu.gt_device_status(sp) == GT_OK
    finally:
        g.set_gram_path(old)
    for k in before:
        assert torch.equal(before[k].view(torch.int32), after[k].view(torch.int32)), k
