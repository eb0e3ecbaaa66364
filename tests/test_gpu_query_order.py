"""The counting sort of queries by leaf: a permutation that visits the leaves' bins in order,
whatever the ratio of queries to points."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nq", [(1, 1), (1, 5000), (17, 3), (100000, 1), (100000, 4097), (5000, 70001)])
@pytest.mark.parametrize("d", [1, 3, 8])
def test_gpu_query_order(gpu, n, nq, d):
    import torch
    from cosmokdtree_b200 import _lib
    rng = np.random.default_rng(n + nq)
    P, Q = rng.random((n, d)), rng.random((nq, d))
    t = gpu.kdtree.build_kdtree(P)
    q = torch.from_numpy(Q).cuda()
    o = torch.empty(nq, dtype=torch.int32, device="cuda")
    _lib.check(_lib.load().ckd_query_order(t.handle, ctypes.c_void_p(q.data_ptr()), nq,
                                           ctypes.c_void_p(o.data_ptr()), None))
    order = o.cpu().numpy()
    np.testing.assert_array_equal(np.sort(order), np.arange(nq))
    e = t.export()
    node = np.zeros(nq, np.int64)  # the leaf of every query, by the split rule
    while True:
        inner = e["axis"][node] >= 0
        if not inner.any():
            break
        a, s = e["axis"][node], e["split"][node]
        left = Q[np.arange(nq), np.maximum(a, 0)] < s
        node = np.where(inner, np.where(left, e["left"][node], e["right"][node]), node)
    shift = 0
    while (n >> (shift + 1)) >= max(nq, 4096):
        shift += 1
    bins = e["start"][node[order]] >> shift
    assert np.all(np.diff(bins) >= 0)
