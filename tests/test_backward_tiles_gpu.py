"""The Pearson adjoint's operand kernels at the edges of their 64 x 64 tiles: within
the f16x3 tolerance of the FP64 oracle, and the same bits whether the gradient's
rows are on 16-byte boundaries (16-byte loads) or not."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def adjoint(lib, X, dG):
    import torch
    p, n = X.shape
    dX = torch.from_numpy(X).cuda()
    out = torch.empty_like(dX)
    vp = lambda t: ctypes.c_void_p(t.data_ptr())
    st = lib.gt_cor_backward_device(vp(dX), p, n, vp(dG), vp(out),
                                    ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert st == 0, lib.gt_last_error().decode()
    torch.cuda.synchronize()
    return out.cpu().numpy()


@pytest.mark.parametrize("p,n", [(64, 33), (65, 31), (124, 40), (130, 65), (192, 32), (321, 7)])
def test_adjoint(gpu, oracle_mod, p, n):
    import torch
    rng = np.random.default_rng(p)
    X = rng.standard_normal((p, n)).astype(np.float32)
    G = (rng.standard_normal((p, p)) * np.exp2(rng.integers(-3, 4, (p, 1)))).astype(np.float32)
    got = adjoint(gpu, X, torch.from_numpy(G).cuda())
    off = torch.empty(p * p + 1, device="cuda")[1:].copy_(torch.from_numpy(G.ravel()))
    assert np.array_equal(got, adjoint(gpu, X, off))
    want = oracle_mod.cor_backward(X, G.astype(np.float64))
    assert np.abs(got - want).max() <= 2e-5 * np.abs(want).max()
