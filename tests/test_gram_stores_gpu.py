"""The Pearson Gram's 16-byte output stores (rows on 16-byte boundaries) against
its 4-byte ones (the same call with outputs 4 bytes off): the same bits, in
both kinds of problem, with ragged last blocks and with outputs left out."""
import ctypes

import pytest

pytestmark = pytest.mark.gpu


def call(lib, A, B, offset, which):
    import torch
    nA, n = A.shape
    nB = B.shape[0]
    outs = [torch.full((nA * nB + 8,), -7.0, device="cuda") if k in which else None for k in range(3)]
    vp = lambda t, o=0: ctypes.c_void_p(t.data_ptr() + 4 * o) if t is not None else None
    st = lib.gt_pmcc_device(0, vp(A), nA, vp(B), nB, n, *[vp(o, offset) for o in outs],
                            ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert st == 0, lib.gt_last_error().decode()
    for o in outs:  # nothing outside the matrix
        if o is not None:
            assert bool((o[:offset] == -7).all()) and bool((o[offset + nA * nB:] == -7).all())
    return [None if o is None else o[offset:offset + nA * nB] for o in outs]


@pytest.mark.parametrize("path", ["f16x3", "f16x6", "bf16x3"])
@pytest.mark.parametrize("nA,nB", [(1764, 0), (2052, 0), (3000, 0), (1300, 2404), (2403, 1284)])
@pytest.mark.parametrize("which", [(0, 1, 2), (1,), (0, 2)])
def test_same_bits(gpu, path, nA, nB, which):
    import torch
    import gputools_gb300 as g
    gen = torch.Generator(device="cuda").manual_seed(nA)
    A = torch.randn((nA, 70), generator=gen, device="cuda")
    B = torch.randn((nB, 70), generator=gen, device="cuda") if nB else A
    old = g.get_gram_path()
    g.set_gram_path(path)
    try:
        quads, singles = call(gpu, A, B, 4, which), call(gpu, A, B, 1, which)
    finally:
        g.set_gram_path(old)
    for a, b in zip(quads, singles):
        assert a is None or torch.equal(a, b)
