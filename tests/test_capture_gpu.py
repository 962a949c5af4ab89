"""Calls captured into a CUDA graph when the workspace has only what other calls left in
it: scratch that a call can do without must not be allocated then (the capture would be
invalid).  The replayed results are those of the same call made directly."""
import ctypes

import pytest

pytestmark = pytest.mark.gpu

GT_OK = 0
vp = lambda t: ctypes.c_void_p(t.data_ptr()) if t is not None else None


def stream():
    import torch
    return ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)


def replayed(gpu, warm, call, outputs):
    """The outputs of `call` captured after a release of the workspace and `warm`, and
    of the same call made directly."""
    import torch
    gpu.gt_release_workspace()
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        if warm:
            assert warm() == GT_OK, gpu.gt_last_error().decode()
        assert gpu.gt_device_status(stream()) == GT_OK
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=side):
        status = call()
    assert status == GT_OK, gpu.gt_last_error().decode()
    for o in outputs:
        o.fill_(-7.0)
    graph.replay()
    torch.cuda.synchronize()
    got = [o.clone() for o in outputs]
    for o in outputs:
        o.fill_(-7.0)
    assert call() == GT_OK, gpu.gt_last_error().decode()
    assert gpu.gt_device_status(stream()) == GT_OK
    return got, outputs


def values(*shape, seed=1):
    import torch
    gen = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randn(shape, generator=gen, device="cuda")


def pearson(gpu, A, B, out):
    n = A.shape[1]
    return lambda: gpu.gt_pmcc_device(0, vp(A), A.shape[0], vp(B), B.shape[0], n, None, vp(out),
                                      None, stream())


@pytest.mark.parametrize("path", ["f16x3", "f16x6"])
def test_pearson_in_pieces(gpu, path):
    """Few tiles of many observations after a problem of many tiles."""
    import torch
    import gputools_gb300 as g
    big, few = values(3000, 2048), values(700, 2048, seed=2)
    bout, out = torch.empty(3000, 3000, device="cuda"), torch.empty(700, 700, device="cuda")
    old = g.get_gram_path()
    g.set_gram_path(path)
    try:
        got, want = replayed(gpu, pearson(gpu, big, big, bout), pearson(gpu, few, few, out), [out])
    finally:
        g.set_gram_path(old)
    # both within the path's tolerance (the sums are cut differently)
    assert float((got[0] - want[0]).abs().max()) <= (3e-7 if path == "f16x6" else 2.2e-5)


def test_small_pearson_of_two_sets(gpu):
    """Both sets' rows go to one buffer, which is too small for the two."""
    import torch
    A0, B0 = values(200, 1000), values(20000, 1000)
    A, B = values(300, 700, seed=2), values(1000, 700, seed=3)
    o0, out = torch.empty(200, 20000, device="cuda"), torch.empty(300, 1000, device="cuda")
    got, want = replayed(gpu, pearson(gpu, A0, B0, o0), pearson(gpu, A, B, out), [out])
    assert float((got[0] - want[0]).abs().max()) <= 1.3e-5


@pytest.mark.parametrize("mds", [True, False])
def test_distance_adjoint(gpu, mds):
    """20000 points of 16 dimensions: 213 MB of partial sums where 25 MB are at hand.  Both
    kernels sum 20000 terms in float, in another order: 2e-5 of the largest entry."""
    import torch
    n, d = 20000, 16
    Z, zo = values(4000, 1500), torch.empty(4000, 4000, device="cuda")
    X, out = values(n, d, seed=2), torch.empty(n, d, device="cuda")
    loss = torch.empty(1, dtype=torch.float64, device="cuda")
    if mds:
        aux = torch.rand(n * (n - 1) // 2, device="cuda") + 4.0
        call = lambda: gpu.gt_mds_stress_device(vp(X), n, d, vp(aux), vp(out), vp(loss), stream())
    else:
        aux = values(n, n, seed=3)
        call = lambda: gpu.gt_dist_backward_device(vp(X), n, d, vp(aux), vp(out), stream())
    got, want = replayed(gpu, pearson(gpu, Z, Z.clone(), zo), call, [out, loss])
    assert float((got[0] - want[0]).abs().max()) <= 2e-5 * float(want[0].abs().max())
    if mds:
        assert abs(float(got[1] - want[1])) <= 1e-6 * float(want[1])


def test_kendall(gpu):
    """100 MB of signs where 34 are at hand: more passes, the same integers."""
    import torch
    n = 1000
    X0, X = values(60, n), values(200, n, seed=2)
    o0 = torch.empty(60, 60, dtype=torch.float64, device="cuda")
    out = torch.empty(200, 200, dtype=torch.float64, device="cuda")
    call = lambda X, o: lambda: gpu.gt_kendall_device(vp(X), X.shape[0], vp(X), X.shape[0], n,
                                                      vp(o), stream())
    got, want = replayed(gpu, call(X0, o0), call(X, out), [out])
    assert torch.equal(got[0], want[0])


@pytest.mark.parametrize("n,d", [(300, 5), (200, 70)])
def test_canberra_as_the_first_call(gpu, n, d):
    import torch
    P = values(n, d).abs()
    P[torch.rand(n, d, device="cuda") < 0.3] = 0
    out = torch.empty(n, n, device="cuda")
    call = lambda: gpu.gt_distances_device(vp(P), n, d, vp(out), 0, 3, ctypes.c_float(2.0), stream())
    got, want = replayed(gpu, None, call, [out])
    assert torch.equal(got[0].view(torch.int32), want[0].view(torch.int32))
