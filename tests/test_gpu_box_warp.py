"""The warp-per-box kernel against the oracle where its shortcuts could differ from the strict
descent: points on box faces and split planes (lattices), whole subtrees, inverted, infinite
and empty boxes, deep and tiny trees.  Offsets and ids are whole numbers, compared for equality
and in order."""
import numpy as np
import pytest

from test_gpu_parity import make_points

pytestmark = pytest.mark.gpu

CASES = [
    # name, n, d, periodic, leaf, nb
    ("tiny", 5, 3, False, 16, 20),
    ("uniform3d", 65, 3, False, 16, 50),
    ("lattice", 20000, 3, False, 16, 400),
    ("lattice_periodic", 20000, 3, True, 1, 400),
    ("lattice_d2", 5000, 2, False, 4, 400),
    ("clustered_dup", 30000, 3, False, 40, 200),
    ("periodic_clustered", 30000, 3, True, 8, 200),
    ("d1", 3000, 1, False, 16, 100),
    ("d5_lattice", 6000, 5, False, 16, 100),
    ("d8", 3000, 8, True, 16, 50),
]


@pytest.mark.parametrize("name,n,d,periodic,leaf,nb", CASES)
def test_gpu_box_warp_matches_oracle(gpu, oracle, name, n, d, periodic, leaf, nb):
    P = make_points(name, n, d, periodic)
    rng = np.random.default_rng(47)
    lo = rng.random((nb, d)) * 1.2 - (0.6 if periodic or "lattice" in name else 0.1)
    hi = lo + rng.choice([0.05, 0.3, 0.9], (nb, 1)) * rng.random((nb, d))
    if "lattice" in name:  # faces on the points' own coordinates, and on the split planes
        half = nb // 2
        lo[:half] = rng.integers(-9, 9, (half, d)) / 16.0
        hi[:half] = lo[:half] + rng.integers(0, 9, (half, d)) / 16.0
    B = np.empty((nb, 2 * d))
    B[:, 0::2], B[:, 1::2] = lo, hi
    B[0, 0::2], B[0, 1::2] = -np.inf, np.inf      # everything
    B[1, 0::2], B[1, 1::2] = P.min(0), P.max(0)   # the tight box: faces on points
    B[2, 0::2], B[2, 1::2] = 0.3, 0.1             # inverted
    B[3, 0::2], B[3, 1::2] = 50.0, 60.0           # outside
    B[4, 0::2] = B[4, 1::2] = P[0]                # one point
    t = gpu.kdtree.build_kdtree(P, leaf=leaf, boxsize=1.0 if periodic else None)
    oo, oi = oracle.OracleTree(P, leaf, 1.0 if periodic else None).box_csr(B)
    xo, xi = (x.cpu().numpy() for x in gpu.kdtree.box_search_csr(t, B))
    np.testing.assert_array_equal(xo, oo)
    np.testing.assert_array_equal(xi, oi)


def test_gpu_box_whole_ranges_as_tasks(gpu):
    """Boxes over everything need more emission tasks than their buffer holds."""
    import torch
    n, nb = 300000, 900  # 74 tasks of 4096 points a row: 66600 tasks against 65536
    rng = np.random.default_rng(5)
    t = gpu.kdtree.build_kdtree(torch.from_numpy(rng.random((n, 3))).cuda())
    B = torch.tensor([[-1.0, 2.0] * 3], dtype=torch.float64, device="cuda").repeat(nb, 1)
    off, idx = gpu.kdtree.box_search_csr(t, B)
    idx = idx.reshape(nb, n)
    assert torch.equal(off, torch.arange(nb + 1, device="cuda") * n)
    assert torch.equal(idx[0].sort().values, torch.arange(n, device="cuda"))
    assert bool((idx == idx[0]).all())


def test_gpu_box_fill_without_room_for_tasks(gpu):
    """With the pool capped at what it holds, the fill copies whole ranges itself."""
    import torch
    from cosmokdtree_b200 import _lib
    L = _lib.load()
    rng = np.random.default_rng(6)
    P = torch.from_numpy(rng.random((300000, 3))).cuda()
    t = gpu.kdtree.build_kdtree(P)
    B = torch.tensor([[0.1, 0.9] * 3, [-1.0, 2.0] * 3, [0.4, 0.45] * 3], dtype=torch.float64,
                     device="cuda")
    want = gpu.kdtree.box_search_csr(t, B)
    _lib.check(L.ckd_set_tuning(9, 1))  # 1 MiB, less than the tree itself holds
    try:
        got = gpu.kdtree.box_search_csr(t, B)
    finally:
        _lib.check(L.ckd_set_tuning(9, 0))
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
