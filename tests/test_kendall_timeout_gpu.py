"""The bounded-wait abort path of Kendall's sign Gram: with a 2 us limit its waits give up
while copies and multiplies are in flight; the block must wait for those, free its
tensor memory and report, and the next call must be exact again."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GT_OK, GT_ETIMEOUT = 0, 5


@pytest.mark.parametrize("nx,ny,n", [(700, 0, 500), (300, 500, 600)])
def test_short_wait_limit_reports_timeout_and_recovers(gpu, oracle_mod, rng, nx, ny, n):
    import torch
    X = rng.integers(0, 10, (nx, n)).astype(np.float32)
    Y = rng.integers(0, 10, (ny, n)).astype(np.float32) if ny else X
    ny = ny or nx
    dX = torch.from_numpy(X).cuda()
    dY = dX if Y is X else torch.from_numpy(Y).cuda()
    out = torch.empty((ny, nx), dtype=torch.float64, device="cuda")
    host = np.empty((ny, nx))
    vp = lambda t: ctypes.c_void_p(t.data_ptr())
    hv = lambda a: a.ctypes.data_as(ctypes.c_void_p)
    sp = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    call = lambda: gpu.gt_kendall_device(vp(dX), nx, vp(dY), ny, n, vp(out), sp)
    assert gpu.gt_device_status(sp) == GT_OK  # nothing pending from earlier tests
    seen = set()
    try:
        assert gpu.gt_set_wait_limit_ns(2000) == GT_OK
        for _ in range(3):
            assert call() == GT_OK, gpu.gt_last_error().decode()
            seen.add(gpu.gt_device_status(sp))
            assert gpu.gt_device_status(sp) == GT_OK  # the check clears the word
        host_status = gpu.gt_kendall(hv(X), nx, hv(Y), ny, n, hv(host))
    finally:
        gpu.gt_set_wait_limit_ns(0)
    assert seen == {GT_ETIMEOUT}, "a 2 us limit never gave up a wait"
    assert host_status == GT_ETIMEOUT, gpu.gt_last_error().decode()
    assert call() == GT_OK
    assert gpu.gt_device_status(sp) == GT_OK
    want, *_ = oracle_mod.kendall(X, Y) if Y is not X else oracle_mod.kendall(X)
    assert np.array_equal(out.cpu().numpy(), want)
