"""Distance adjoint and MDS stress with NaN coordinates: a pair with one adds nothing to
the gradient, so only the NaN coordinates' own entries are NaN, whichever tile their point
is in (an infinity still reaches every point)."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

U = 2.0 ** -24


def run(lib, X, aux, mode):
    import torch
    n, d = X.shape
    dX, da = torch.from_numpy(X).cuda(), torch.from_numpy(aux).cuda()
    out = torch.full((n, d), 7.0, device="cuda")
    loss = torch.zeros(1, dtype=torch.float64, device="cuda")
    vp = lambda t: ctypes.c_void_p(t.data_ptr())
    s = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    if mode == "mds":
        st = lib.gt_mds_stress_device(vp(dX), n, d, vp(da), vp(out), vp(loss), s)
    else:
        st = lib.gt_dist_backward_device(vp(dX), n, d, vp(da), vp(out), s)
    assert st == 0, lib.gt_last_error().decode()
    return out.cpu().numpy(), float(loss.item())


def inputs(rng, n, d, mode):
    X = rng.standard_normal((n, d)).astype(np.float32)
    if mode == "mds":
        return X, (rng.random(n * (n - 1) // 2) * 3 + 0.5).astype(np.float32)
    return X, rng.standard_normal((n, n)).astype(np.float32)


@pytest.mark.parametrize("mode", ["mds", "dist"])
@pytest.mark.parametrize("n,d,bad", [(2, 2, [0]), (65, 3, [64]), (129, 16, [3, 128]), (193, 17, [63, 64]),
                                     (300, 40, [0, 130, 131, 299]), (1600, 32, [77, 800])])
def test_nan_coordinates(gpu, rng, mode, n, d, bad):
    X, aux = inputs(rng, n, d, mode)
    for k, i in enumerate(bad):
        X[i, (5 * k) % d] = np.nan
    grad, loss = run(gpu, X, aux, mode)
    P = X.astype(np.float64)
    D = np.sqrt(sum((P[:, None, k] - P[None, :, k]) ** 2 for k in range(d)))
    off = ~np.eye(n, dtype=bool)
    live = off & ~np.isnan(D)
    D1 = np.where(live, D, 1.0)
    if mode == "mds":
        T = np.ones((n, n))
        j, i = np.triu_indices(n, 1)
        T[i, j] = T[j, i] = aux
        E = np.where(np.isnan(D), 0.0, D) - T
        W = np.where(live, 2 * E / D1, 0.0)
        # D within 4 roundings, its square's term and the sum within 3
        bound = 0.5 * U * (8 * np.abs(E) * D1 + 3 * E * E)[off].sum()
        assert abs(loss - 0.5 * (E * E)[off].sum()) <= bound
        A = np.where(live, np.abs(W) + 2, 0.0)
    else:
        W = np.where(live, (aux + aux.T).astype(np.float64) / D1, 0.0)
        A = np.abs(W)
    V = np.nan_to_num(P)  # (pairs with a NaN have W = 0)
    want = V * W.sum(1, keepdims=True) - W @ V
    nan = np.isnan(P)
    assert np.array_equal(np.isnan(grad), nan)
    # every term rounded 110 times at most
    tol = 110 * U * (A.sum(1, keepdims=True) * np.abs(V) + A @ np.abs(V))
    assert np.all(np.abs(grad - want)[~nan] <= tol[~nan])


@pytest.mark.parametrize("mode", ["mds", "dist"])
def test_an_infinite_coordinate_reaches_every_point(gpu, rng, mode):
    X, aux = inputs(rng, 150, 8, mode)
    X[70, 3] = np.inf
    grad, _ = run(gpu, X, aux, mode)
    assert np.all(np.isnan(grad[:, 3]))
    if mode == "dist":  # W = G / Inf = 0: the other coordinates stay finite
        assert np.all(np.isfinite(np.delete(grad, 3, axis=1)))
