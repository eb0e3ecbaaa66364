"""The warp-per-query ball kernel against the oracle at the edges of its scan units, its batch
rule and its hand-overs.  Counts, ids and FP64 distances are compared for equality (separately
rounded arithmetic on both sides); unsorted periodic rows hold the reference's points in leaf
order, so they are compared sorted."""
import numpy as np
import pytest

from test_gpu_parity import make_points

pytestmark = pytest.mark.gpu

CASES = [
    # name, n, d, periodic, leaf, nq, r
    ("tiny", 5, 3, False, 16, 3, 0.4),
    ("uniform3d", 65, 3, False, 16, 9, 0.3),            # one scan unit past the root's
    ("uniform3d", 6000, 3, False, 16, 33, 0.05),
    ("periodic3d", 6000, 3, True, 8, 33, 0.2),          # balls across the faces
    ("periodic_clustered", 20000, 3, True, 16, 64, 0.45),
    ("clustered_dup", 20000, 3, False, 40, 64, 0.02),   # leaves longer than a unit
    ("lattice", 8000, 3, False, 1, 40, 0.125),          # distances equal to the radius
    ("lattice_periodic", 8000, 3, True, 16, 40, 0.25),
    ("d1", 3000, 1, True, 16, 17, 0.01),
    ("d2", 3000, 2, False, 3, 17, 0.1),
    ("d5", 3000, 5, False, 16, 17, 0.4),
    ("d8", 3000, 8, True, 16, 17, 0.6),
]


@pytest.mark.parametrize("sorted_", [False, True])
@pytest.mark.parametrize("name,n,d,periodic,leaf,nq,r", CASES)
def test_gpu_ball_warp_matches_oracle(gpu, oracle, name, n, d, periodic, leaf, nq, r, sorted_):
    P = make_points(name, n, d, periodic)
    rng = np.random.default_rng(41)
    Q = np.concatenate([P[rng.integers(0, n, nq // 2)],
                        rng.random((nq - nq // 2, d)) - (0.5 if periodic else 0.0)])
    if not periodic:
        Q[-1] = 1e30  # far beyond FP32 squares
    box = 1.0 if periodic else None
    t = gpu.kdtree.build_kdtree(P, leaf=leaf, boxsize=box)
    ooff, oidx, odist = oracle.OracleTree(P, leaf, box).ball_csr(Q, r, sorted=sorted_)
    off, idx, dist = (x.cpu().numpy() for x in
                      gpu.kdtree.ball_search_csr(t, Q, r, sorted=sorted_))
    np.testing.assert_array_equal(off, ooff)
    if sorted_ or not periodic:
        np.testing.assert_array_equal(idx, oidx)
        np.testing.assert_array_equal(dist, odist)
    else:
        for a, b in zip(off[:-1], off[1:]):
            np.testing.assert_array_equal(np.sort(idx[a:b]), np.sort(oidx[a:b]))
            np.testing.assert_array_equal(np.sort(dist[a:b]), np.sort(odist[a:b]))


@pytest.mark.parametrize("sorted_", [False, True])
@pytest.mark.parametrize("name,d,periodic,leaf,nq,hits", [
    ("uniform3d", 3, False, 16, 11999, 4.0),   # below the eight lanes' batch
    ("uniform3d", 3, False, 16, 12001, 4.0),   # eight lanes per query
    ("uniform3d", 3, False, 1, 12001, 15.9),
    ("uniform3d", 3, False, 16, 12001, 16.1),  # past their result count
    ("uniform3d", 3, True, 40, 12003, 10.0),   # across the faces, leaves past a unit
    ("lattice", 3, False, 16, 12001, 8.0),
    ("lattice_periodic", 2, True, 16, 12001, 8.0),
    ("d1", 1, True, 16, 12001, 3.0),
    ("d5", 5, False, 16, 12001, 2.0),
    ("uniform3d", 3, False, 16, 100001, 60.0),
])
def test_gpu_ball_eight_lanes(gpu, oracle, name, d, periodic, leaf, nq, hits, sorted_):
    n = 20000
    P = make_points(name, n, d, periodic)
    rng = np.random.default_rng(53)
    Q = np.concatenate([P[rng.integers(0, n, nq // 2)],
                        rng.random((nq - nq // 2, d)) - (0.5 if periodic else 0.0)])
    if not periodic:
        Q[-1] = np.nan
        Q[-2] = -1e40
    side = 1.0 if periodic else P.max(0) - P.min(0)
    ball = [0, 2.0, 3.14159, 4.18879, 0, 5.26379][d]
    r = float((hits / (n * ball) * np.prod(np.broadcast_to(side, d))) ** (1.0 / d))
    box = 1.0 if periodic else None
    t = gpu.kdtree.build_kdtree(P, leaf=leaf, boxsize=box)
    ooff, oidx, odist = oracle.OracleTree(P, leaf, box).ball_csr(Q, r, sorted=sorted_)
    off, idx, dist = (x.cpu().numpy() for x in
                      gpu.kdtree.ball_search_csr(t, Q, r, sorted=sorted_))
    np.testing.assert_array_equal(off, ooff)
    if sorted_ or not periodic:
        np.testing.assert_array_equal(idx, oidx)
        np.testing.assert_array_equal(dist, odist)
    else:
        for a, b in zip(off[:-1][::7], off[1:][::7]):
            np.testing.assert_array_equal(np.sort(idx[a:b]), np.sort(oidx[a:b]))


@pytest.mark.parametrize("name,r", [("uniform3d", 0.01), ("clustered_deep", 0.004)])
def test_gpu_ball_batches_past_the_warp_rule(gpu, name, r):
    """A batch past the rule (packets first, heavy ones handed over on an uneven tree) gives
    the rows of the same queries in small batches."""
    rng = np.random.default_rng(43)
    n, nq = 410000, 200001
    P = rng.random((n, 3))
    if name == "clustered_deep":  # most points in a few very dense clumps
        c = rng.random((6, 3))
        P[: n - 20000] = c[rng.integers(0, 6, n - 20000)] + \
            rng.standard_normal((n - 20000, 3)) * 10.0 ** rng.uniform(-6, -2, (n - 20000, 1))
    t = gpu.kdtree.build_kdtree(P)
    Q = P[rng.integers(0, n, nq)]
    if name == "clustered_deep":
        Q[: nq - 2000] = rng.random((nq - 2000, 3)) * 3.0  # mostly empty rows, some very long
    off, idx, dist = gpu.kdtree.ball_search_csr(t, Q, r)
    ids = rng.integers(0, nq, 3000)
    ids[:500] = nq - 1 - np.arange(500)
    soff, sidx, sdist = gpu.kdtree.ball_search_csr(t, Q[ids], r)
    off, soff = off.cpu().numpy(), soff.cpu().numpy()
    np.testing.assert_array_equal(np.diff(off)[ids], np.diff(soff))
    take = np.concatenate([np.arange(off[i], off[i + 1]) for i in ids])
    np.testing.assert_array_equal(idx.cpu().numpy()[take], sidx.cpu().numpy())
    np.testing.assert_array_equal(dist.cpu().numpy()[take], sdist.cpu().numpy())


def sampled_rows_match(search, batch, sample, ids, nq):
    """Rows ``ids`` of a large batch equal the same queries searched in small ones."""
    off, idx, dist = (x.cpu().numpy() for x in search(batch))
    soff, sidx, sdist = (x.cpu().numpy() for x in search(sample))
    assert len(off) == nq + 1 and soff[-1] > 0
    np.testing.assert_array_equal(np.diff(off)[ids], np.diff(soff))
    take = np.concatenate([np.arange(off[i], off[i + 1]) for i in ids])
    np.testing.assert_array_equal(idx[take], sidx)
    np.testing.assert_array_equal(dist[take], sdist)


@pytest.mark.parametrize("sorted_", [False, True])
def test_gpu_ball_packets_on_deep_trees(gpu, sorted_):
    """Packets of a batch past the warp rule on a tree deeper than their shared stack
    (96 entries): a cusp at a low corner, whose leftmost paths keep a sibling a level."""
    rng = np.random.default_rng(61)
    n, nq = 400001, 200001
    P = rng.random((n, 3)) * 10.0 ** (-10 * rng.random((n, 1)))
    t = gpu.kdtree.build_kdtree(P)
    assert 96 <= t.depth < 127
    near = np.argsort((P * P).sum(1))[:nq]  # the deepest leaves are all among them
    Q = P[near]
    ids = np.concatenate([np.arange(2000), rng.integers(2000, nq, 2000)])
    sampled_rows_match(lambda q: gpu.kdtree.ball_search_csr(t, q, 1e-11, sorted=sorted_),
                       Q, Q[ids], ids, nq)


def test_gpu_ball_packets_on_deep_forests(gpu):
    """The same in a forest, where the packets hold several roots besides."""
    rng = np.random.default_rng(67)
    trees, m, per = 20001, 110, 10
    P = 0.5 ** np.arange(m)[None, :, None] * (1 + 0.1 * rng.random((trees, m, 3)))
    poff = np.arange(trees + 1) * m
    f = gpu.build_forest(P.reshape(-1, 3), poff, leaf=1)
    assert 96 <= f.depth < 127
    Q = P[:, m - per:]  # next to the corner of each tree
    pick = np.arange(0, trees, 97)
    ids = (pick[:, None] * per + np.arange(per)).ravel()

    def search(q):
        return f.ball_csr(q.reshape(-1, 3), qoff[len(q)], 1e-31)

    qoff = {trees: np.arange(trees + 1) * per}
    few = np.zeros(trees + 1, np.int64)
    few[pick + 1] = per
    qoff[len(pick)] = np.cumsum(few)
    sampled_rows_match(search, Q, Q[pick], ids, trees * per)


@pytest.mark.parametrize("periodic", [False, True])
def test_gpu_ball_kernels_of_a_loaded_tree(gpu, tmp_path, periodic):
    """A tree read back from its file is searched by the kernels that the built one is: the
    same rows in as many launches (eight lanes a query need one fewer than a warp)."""
    from cosmokdtree_b200 import _lib
    L = _lib.load()
    rng = np.random.default_rng(79)
    P = rng.random((20000, 3)) - 0.5
    t = gpu.kdtree.build_kdtree(P, boxsize=1.0 if periodic else None)
    gpu.kdtree.save_kdtree(t, str(tmp_path / "tree"))
    u = gpu.kdtree.load_kdtree(str(tmp_path / "tree"))

    def run(tree):
        before = L.ckd_launch_count()
        out = [x.cpu().numpy() for x in gpu.kdtree.ball_search_csr(tree, P[:12001], 0.03)]
        return out, L.ckd_launch_count() - before

    (a, na), (b, nb) = run(t), run(u)
    for x, y in zip(a, b):
        np.testing.assert_array_equal(x, y)
    assert na == nb


@pytest.mark.parametrize("n,nq,hits", [
    (1 << 18, 200001, 130), (1 << 18, 200001, 220), (10000, 100001, 20), (10000, 100001, 200)])
def test_gpu_ball_rows_on_both_sides_of_the_packets_line(gpu, n, nq, hits):
    """Even trees: short and long rows in one batch, on both sides of the mean that decides, and
    the line of small trees, against the same queries in small batches."""
    rng = np.random.default_rng(89)
    P = rng.random((n, 3))
    t = gpu.kdtree.build_kdtree(P)
    Q = P[rng.integers(0, n, nq)]
    r = float((hits / (n * 4.18879)) ** (1 / 3))
    ids = rng.integers(0, nq, 3000)
    sampled_rows_match(lambda q: gpu.kdtree.ball_search_csr(t, q, r), Q, Q[ids], ids, nq)


def test_gpu_ball_packets_fill_the_short_rows_of_even_trees(gpu):
    """3 x 10^5 rows of some 80 results on an even tree: the fill takes at most twice as long as
    the count (1.4 times with packets; a warp a row took 2.7 times)."""
    import ctypes
    import torch
    from cosmokdtree_b200 import _lib
    L = _lib.load()
    g = torch.Generator(device="cuda")
    g.manual_seed(3)
    n, nq = 1 << 20, 300000
    P = torch.rand(n, 3, generator=g, device="cuda", dtype=torch.float64)
    Q = P[torch.arange(nq, device="cuda") * 7919 % n].contiguous()
    r = float((80 / (n * 4.18879)) ** (1 / 3))
    t = gpu.kdtree.build_kdtree(P)
    off, idx, dist = gpu.kdtree.ball_search_csr(t, Q, r)
    counts = torch.empty(nq, dtype=torch.int64, device="cuda")
    ptr = lambda x: ctypes.c_void_p(x.data_ptr())
    s = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)

    def clock(f):
        best = np.inf
        for _ in range(8):
            a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            a.record()
            _lib.check(f())
            b.record()
            torch.cuda.synchronize()
            best = min(best, a.elapsed_time(b))
        return best

    tc = clock(lambda: L.ckd_ball_count(t.handle, ptr(Q), nq, r, ptr(counts), s))
    tf = clock(lambda: L.ckd_ball_fill_sized(t.handle, ptr(Q), nq, r, 0, int(off[-1]), ptr(off),
                                             ptr(idx), ptr(dist), s))
    print("count %.3f fill %.3f ms" % (tc, tf))
    assert tf < 2.0 * tc
