"""Clustering where merged-away columns may not be skipped (infinite entries of an
asymmetric matrix), and at the sizes where the threads of a CTA and the columns
that a thread owns change: merges, order and heights are the oracle's."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

METHODS = ["single", "complete", "average", "mcquitty", "wpgma", "median", "centroid",
           "flexible", "flexible_group", "ward"]


def check(lib, oracle_mod, D, method):
    n = D.shape[0]
    merge, order = np.empty(2 * (n - 1), np.int32), np.empty(n, np.int32)
    height = np.empty(n - 1, np.float32)
    D = np.ascontiguousarray(D, np.float32)
    vp = lambda a: a.ctypes.data_as(ctypes.c_void_p)
    assert lib.gt_hclust(vp(D), n, method.encode(), vp(merge), vp(order), vp(height)) == 0
    sub, sup, val = oracle_mod.hclust(D, method)
    m2, o2 = oracle_mod.format_clustering(sub, sup)
    np.testing.assert_array_equal(merge.reshape(2, n - 1).T, m2)
    np.testing.assert_array_equal(order, o2)
    np.testing.assert_array_equal(height.view(np.int32), np.asarray(val, np.float32).view(np.int32))


@pytest.mark.parametrize("method", METHODS)
def test_infinite_entries(gpu, oracle_mod, method):
    rng = np.random.default_rng(31)
    D = rng.random((150, 150)).astype(np.float32)
    D[3, 100:104] = np.inf  # row 3 only, not column 3; every merge stays finite
    np.fill_diagonal(D, 0)
    check(gpu, oracle_mod, D, method)


@pytest.mark.parametrize("ctas,n", [("1", 128), ("1", 129), ("1", 257), ("1", 512), ("1", 513),
                                    ("2", 1024), ("2", 1025)])
def test_threads_and_columns(gpu, oracle_mod, monkeypatch, ctas, n):
    monkeypatch.setenv("GT_HCLUST_CTAS", ctas)
    rng = np.random.default_rng(n)
    P = rng.standard_normal((n, 3)).astype(np.float32)
    D = np.abs(P[:, None] - P[None]).max(-1)
    for method in ("average", "complete", "median"):
        check(gpu, oracle_mod, D, method)
