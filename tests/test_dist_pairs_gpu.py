"""The distance adjoint over unordered pairs of 64 x 64 tiles: edges of the tiles
and of the three dimension classes, rows off the 16-byte boundaries, segments
that end inside and at the end of a row of tiles, and coincident points."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


U = 2.0 ** -24


def distances(X):
    """FP64 distances of the float points (direct differences), 1 on the diagonal."""
    P = X.astype(np.float64)
    D = np.sqrt(sum((P[:, None, k] - P[None, :, k]) ** 2 for k in range(P.shape[1])))
    np.fill_diagonal(D, 1.0)
    return D


def grad_bound(X, W):
    """Componentwise: x_i sum_j W_ij - sum_j W_ij x_j rounds each term at most 110
    times (64 in a tile, the tiles of a segment, the partial sums, and W itself)."""
    A, V = np.abs(W), np.abs(X.astype(np.float64))
    np.fill_diagonal(A, 0.0)
    return 110 * U * (A.sum(1, keepdims=True) * V + A @ V)


def points(rng, n, d):
    X = rng.standard_normal((n, d)).astype(np.float32)
    if n > 20:
        X[n - 3] = X[4]
        X[7] = X[6]
    return X


def run(lib, X, aux, mode, offset):
    import torch
    n, d = X.shape
    buf = torch.zeros(n * d + offset, device="cuda")
    buf[offset:] = torch.from_numpy(X.ravel()).cuda()
    da = torch.from_numpy(aux).cuda()
    out = torch.full((n, d), float("nan"), device="cuda")
    loss = torch.zeros(1, dtype=torch.float64, device="cuda")
    vp = lambda t, o=0: ctypes.c_void_p(t.data_ptr() + 4 * o)
    s = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    if mode == "mds":
        st = lib.gt_mds_stress_device(vp(buf, offset), n, d, vp(da), vp(out), vp(loss), s)
    else:
        st = lib.gt_dist_backward_device(vp(buf, offset), n, d, vp(da), vp(out), s)
    assert st == 0, lib.gt_last_error().decode()
    return out.cpu().numpy().astype(np.float64), float(loss.item())


SHAPES = [(2, 1), (3, 2), (63, 15), (64, 16), (65, 17), (127, 31), (129, 32), (200, 33), (193, 63),
          (256, 64), (1500, 3), (1601, 20)]


@pytest.mark.parametrize("n,d", SHAPES)
@pytest.mark.parametrize("offset", [0, 1])
def test_mds_stress(gpu, oracle_mod, rng, n, d, offset):
    X = points(rng, n, d)
    delta = (rng.random(n * (n - 1) // 2) * 3 + 0.5).astype(np.float32)
    grad, loss = run(gpu, X, delta, "mds", offset)
    want_loss, want = oracle_mod.mds_stress(X, delta)
    D = distances(X)
    T = np.ones((n, n))
    j, i = np.triu_indices(n, 1)  # dist order: columns j, rows i > j
    T[i, j] = T[j, i] = delta
    E = D - T
    # D is within 4 roundings, so is each term 2 |E| times as much; its square, the
    # residual and the sum are within 3
    off = ~np.eye(n, dtype=bool)
    assert abs(loss - want_loss) <= 0.5 * U * (8 * np.abs(E) * D + 3 * E * E)[off].sum()
    # W = 2 E / D: the error of D counts as 2 at most
    assert np.all(np.abs(grad - want) <= grad_bound(X, 2 * np.abs(E) / np.where(D > 0, D, 1.0) + 2))


@pytest.mark.parametrize("n,d", SHAPES)
def test_distance_adjoint(gpu, oracle_mod, rng, n, d):
    X = points(rng, n, d)
    G = rng.standard_normal((n, n)).astype(np.float32)
    grad, _ = run(gpu, X, G, "dist", 0)
    want = oracle_mod.dist_backward(X, G.astype(np.float64))
    D = distances(X)
    assert np.all(np.abs(grad - want) <= grad_bound(X, np.where(D > 0, (G + G.T) / np.where(D > 0, D, 1.0), 0.0)))


def test_repeated_calls_agree(gpu, rng):
    X = points(rng, 5000, 24)
    delta = (rng.random(5000 * 4999 // 2) * 3 + 0.5).astype(np.float32)
    a, b = run(gpu, X, delta, "mds", 0), run(gpu, X, delta, "mds", 0)
    assert np.array_equal(a[0], b[0]) and a[1] == b[1]
