"""Subtrees built in shared memory (nodes of at most 2048 points for d <= 3, 1024 above) against
the oracle's recursion, at the edges of that size, of the block- and warp-split nodes and of the
leaf size, on slides, duplicates and signed zeros.  Structure, ids and FP64 cells are compared
for equality."""
import numpy as np
import pytest

from test_gpu_parity import clustered, make_points

pytestmark = pytest.mark.gpu


def same_tree(gpu, oracle, P, leaf, box):
    t = gpu.kdtree.build_kdtree(P, leaf=leaf, boxsize=box)
    ot = oracle.OracleTree(P, leaf, box)
    assert t.n_nodes == ot.n_nodes
    g, o = t.export(), ot.export()
    for key in ("axis", "start", "count", "left", "right", "cell", "ids"):
        np.testing.assert_array_equal(g[key], o[key], err_msg=key)
    inner = g["axis"] >= 0
    np.testing.assert_array_equal(g["split"][inner], o["split"][inner])
    pts = o["pts"]
    for a in np.unique(np.r_[0, np.random.default_rng(1).integers(0, t.n_nodes, 200)]):
        seg = pts[g["start"][a]:g["start"][a] + g["count"][a]]
        np.testing.assert_array_equal(seg.min(0), g["box"][a][0::2])
        np.testing.assert_array_equal(seg.max(0), g["box"][a][1::2])
    return t


@pytest.mark.parametrize("n", [1, 2, 16, 17, 33, 511, 512, 513, 1024, 1025, 2047, 2048, 2049, 4097])
@pytest.mark.parametrize("d,periodic", [(3, False), (3, True), (5, False)])
def test_gpu_finish_sizes(gpu, oracle, n, d, periodic):
    P = make_points("uniform", n, d, periodic, seed=n)
    same_tree(gpu, oracle, P, 16, 1.0 if periodic else None)


@pytest.mark.parametrize("leaf", [1, 2, 40, 1023, 1024, 2047, 2048, 3000])
def test_gpu_finish_leaf_sizes(gpu, oracle, leaf):
    same_tree(gpu, oracle, make_points("clustered", 7001, 3, True), leaf, 1.0)
    same_tree(gpu, oracle, make_points("clustered", 5001, 4, False), leaf, None)


@pytest.mark.parametrize("d", [1, 2, 3, 6, 8])
def test_gpu_finish_ties_slides_zeros(gpu, oracle, d):
    rng = np.random.default_rng(7 + d)
    P = rng.integers(-3, 4, (3000, d)) / 8.0          # equal coordinates on every axis
    P[rng.random((3000, d)) < 0.3] = -0.0              # both zeros, the periodic box's midpoint
    P[100:160] = P[100]                                # duplicates peel one point a level
    same_tree(gpu, oracle, P, 64, 1.0)
    same_tree(gpu, oracle, P + 0.0, 64, None)


def test_gpu_finish_more_nodes_than_planned(gpu, oracle):
    """A tree with more nodes than four per full leaf is built with room for all."""
    n = 6000
    P = np.zeros((n, 2))
    P[:, 0] = np.cumsum(1.5 ** -np.arange(n).clip(0, 600)) + np.arange(n) * 1e-12
    P[:, 1] = np.arange(n) % 7
    P[n // 2:] = P[n // 2]                              # 3000 copies of one point
    for leaf in (8, 16):
        t = same_tree(gpu, oracle, P, leaf, None)
        d, i = gpu.kdtree.knn_search(t, P[:50], 5)
        od, oi = oracle.OracleTree(P, leaf, None).knn(P[:50], 5)
        np.testing.assert_array_equal(i, oi)
        np.testing.assert_array_equal(d, od)


def test_gpu_finish_forest(gpu, oracle):
    rng = np.random.default_rng(3)
    sizes = [1, 16, 17, 100, 2048, 2049, 30000, 5]
    parts = [clustered(rng, n, 3, True) for n in sizes]
    f = gpu.build_forest(parts, leaf=16, boxsize=1.0)
    assert f.n_nodes == sum(oracle.OracleTree(P, 16, 1.0).n_nodes for P in parts)
    q = np.concatenate([P[:20] for P in parts])
    qoff = np.cumsum([0] + [min(20, n) for n in sizes])
    d, i = f.knn(q, qoff, 6)
    for t, P in enumerate(parts):
        od, oi = oracle.OracleTree(P, 16, 1.0).knn(P[:20], 6)
        np.testing.assert_array_equal(i[qoff[t]:qoff[t + 1]].cpu().numpy(), oi)
        np.testing.assert_array_equal(d[qoff[t]:qoff[t + 1]].cpu().numpy(), od)


@pytest.mark.parametrize("kind,n,d,leaf", [
    ("copies", 2000, 3, 16),      # one subtree, no levels before it
    ("copies", 60000, 3, 16),     # many subtrees, some of which find room
    ("copies", 60000, 2, 64),     # room several times too small
    ("copies", 40000, 5, 3),
    ("half", 60001, 3, 16),
    ("clumps", 60000, 3, 256),
    ("clumps", 60000, 6, 64),
])
def test_gpu_finish_grows_and_resumes(gpu, oracle, kind, n, d, leaf):
    """Subtrees that found no room for their nodes are finished again, not the whole tree."""
    from cosmokdtree_b200 import _lib
    L = _lib.load()
    rng = np.random.default_rng(71)
    U = rng.random((n, d))
    if kind == "copies":
        P = np.repeat(U[:n // 100], 100, 0)[rng.permutation(n)]
    elif kind == "half":
        P = np.where(np.arange(n)[:, None] % 2, U, U[np.arange(n) // 400 * 400])
    else:
        P = U[rng.integers(0, 40, n)] + 10.0 ** rng.uniform(-9, -1, (n, 1)) * rng.normal(size=(n, d))

    def launches(pts):
        before = L.ckd_launch_count()
        gpu.kdtree.build_kdtree(pts, leaf=leaf)
        return L.ckd_launch_count() - before

    t = same_tree(gpu, oracle, P, leaf, None)
    assert t.n_nodes > 4 * (n // leaf) + 65  # more than planned
    if n == 2000:
        assert launches(P) <= launches(U) + 2  # the even tree's, and k_finish again
    d_, i_ = gpu.kdtree.knn_search(t, P[:50], 5)
    od, oi = oracle.OracleTree(P, leaf, None).knn(P[:50], 5)
    np.testing.assert_array_equal(i_, oi)
    np.testing.assert_array_equal(d_, od)


def test_gpu_finish_grows_and_resumes_in_a_forest(gpu, oracle):
    rng = np.random.default_rng(73)
    parts = [rng.random((n, 3)) for n in (700, 3000, 1, 9000, 50)]
    parts += [np.repeat(rng.random((n // 50, 3)), 50, 0) for n in (3000, 20000, 1000)]
    f = gpu.build_forest(parts, leaf=16)
    assert f.n_nodes == sum(oracle.OracleTree(P, 16, None).n_nodes for P in parts)
    q = np.concatenate([P[:20] for P in parts])
    qoff = np.cumsum([0] + [min(20, len(P)) for P in parts])
    d, i = f.knn(q, qoff, 6)
    for t, P in enumerate(parts):
        od, oi = oracle.OracleTree(P, 16, None).knn(P[:20], 6)
        np.testing.assert_array_equal(i[qoff[t]:qoff[t + 1]].cpu().numpy(), oi)
        np.testing.assert_array_equal(d[qoff[t]:qoff[t + 1]].cpu().numpy(), od)


def test_gpu_finish_grows_within_a_memory_cap(gpu):
    """Where the pool has no room for the most nodes that a tree can have, the arrays grow
    twofold: 2^20 6-D points with 1.2 times the planned nodes are built in 400 MiB."""
    import ctypes
    import torch
    from cosmokdtree_b200 import _lib
    L = _lib.load()
    g = torch.Generator(device="cuda")
    g.manual_seed(1)
    n = 1 << 20
    c = torch.rand(64, 6, generator=g, device="cuda", dtype=torch.float64)
    s = 10 ** (-4 * torch.rand(64, 1, generator=g, device="cuda", dtype=torch.float64) - 1)
    j = torch.randint(0, 64, (n,), generator=g, device="cuda")
    P = torch.remainder(c[j] + s[j] * torch.randn(n, 6, generator=g, device="cuda",
                                                  dtype=torch.float64), 1.0)
    want = gpu.kdtree.build_kdtree(P, leaf=64)
    assert want.n_nodes > 4 * (n // 64) + 65
    used, reserved = ctypes.c_int64(), ctypes.c_int64()
    _lib.check(L.ckd_pool_usage(ctypes.byref(used), ctypes.byref(reserved)))
    _lib.check(L.ckd_set_tuning(9, (used.value >> 20) + 400))
    try:
        t = gpu.kdtree.build_kdtree(P, leaf=64)
    finally:
        _lib.check(L.ckd_set_tuning(9, 0))
    a, b = want.export(), t.export()
    for key in ("axis", "split", "start", "count", "left", "right", "cell", "box", "ids"):
        np.testing.assert_array_equal(a[key], b[key], err_msg=key)
