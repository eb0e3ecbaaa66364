"""Long rows of a fill cut into parts against the same fill with the rows walked whole (the total
of the results not given), itself compared with the oracle elsewhere.  Offsets, ids, their order
and FP64 distances are compared for equality."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def cluster(n, d, seed):
    """Points about one centre with a steep profile: a deep, uneven tree."""
    rng = np.random.default_rng(seed)
    x = rng.normal(size=(n, d))
    return x / np.linalg.norm(x, axis=1, keepdims=True) * 0.4 * rng.random((n, 1)) ** 3


def whole(L, lib, handle, x, offsets, r, sorted_, xoff=None):
    import torch
    ptr = lambda t: ctypes.c_void_p(t.data_ptr())
    total = int(offsets[-1])
    idx = torch.empty(total, dtype=torch.int64, device="cuda")
    dist = torch.empty(total, dtype=torch.float64, device="cuda")
    grp = [] if xoff is None else [ptr(xoff)]
    pre = "ckd_" if xoff is None else "ckd_forest_"
    s = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    if r is None:
        lib.check(getattr(L, pre + "box_fill")(handle, ptr(x), *grp, x.shape[0], ptr(offsets),
                                               ptr(idx), s))
    else:
        lib.check(getattr(L, pre + "ball_fill")(handle, ptr(x), *grp, x.shape[0], r, sorted_,
                                                ptr(offsets), ptr(idx), ptr(dist), s))
    return idx, dist


@pytest.mark.parametrize("d,periodic,leaf,nq,r", [
    (3, False, 16, 1, 0.02),
    (3, True, 16, 300, 0.05),
    (3, False, 1, 4736, 0.001),   # the largest batch
    (3, True, 300, 33, 0.02),     # leaves longer than a scan unit
    (2, False, 16, 100, 0.01),
    (6, False, 32, 65, 0.05),
])
def test_gpu_cut_rows_match_whole(gpu, d, periodic, leaf, nq, r):
    import torch
    from cosmokdtree_b200 import _lib
    L = _lib.load()
    n = 1 << 19
    P = torch.from_numpy(cluster(n, d, 3)).cuda()
    pick = torch.arange(nq, device="cuda") * 7919 % n
    pick[0] = (P * P).sum(1).argmin()  # the longest row
    Q = P[pick].contiguous()
    t = gpu.kdtree.build_kdtree(P, leaf=leaf, boxsize=1.0 if periodic else None)
    for sorted_ in (0, 1):
        off, idx, dist = gpu.kdtree.ball_search_csr(t, Q, r, sorted=bool(sorted_))
        assert int(off[-1]) >= 192 * nq
        widx, wdist = whole(L, _lib, t.handle, Q, off, r, sorted_)
        assert torch.equal(idx, widx) and torch.equal(dist, wdist)
    w = r * torch.linspace(0.3, 1.0, nq, device="cuda", dtype=torch.float64)[:, None]
    B = torch.stack([Q - w, Q + w], 2)
    B[0, :, 0], B[0, :, 1] = P[5], P[5] + r       # a face on a point
    B = B.reshape(nq, 2 * d).contiguous()
    off, idx = gpu.kdtree.box_search_csr(t, B)
    assert torch.equal(idx, whole(L, _lib, t.handle, B, off, None, 0)[0])


def test_gpu_cut_rows_of_a_forest(gpu):
    import torch
    from cosmokdtree_b200 import _lib, forest
    L = _lib.load()
    sizes = [400000, 17, 200000, 3000]
    P = np.concatenate([cluster(m, 3, i) for i, m in enumerate(sizes)])
    off = np.concatenate([[0], np.cumsum(sizes)])
    f = forest.build_forest(torch.from_numpy(P).cuda(), off, leaf=16)
    per = 50
    q = np.concatenate([P[a:b][np.arange(per) * 31 % (b - a)] for a, b in zip(off[:-1], off[1:])])
    qoff = torch.arange(len(sizes) + 1, device="cuda") * per
    Q = torch.from_numpy(q).cuda()
    o, idx, dist = f.ball_csr(Q, qoff.cpu().numpy(), 0.02)
    assert int(o[-1]) >= 192 * len(q)
    wi, wd = whole(L, _lib, f.handle, Q, o, 0.02, 0, qoff)
    assert torch.equal(idx, wi) and torch.equal(dist, wd)
    B = torch.stack([Q - 0.01, Q + 0.01], 2).reshape(-1, 6).contiguous()
    o, idx = f.box_csr(B, qoff.cpu().numpy())
    assert int(o[-1]) >= 192 * len(q)
    assert torch.equal(idx, whole(L, _lib, f.handle, B, o, None, 0, qoff)[0])


@pytest.fixture(scope="module")
def core_forest(gpu):
    """Two deep trees, each with 8192 targets about its dense core: the 16384 rows of thousands
    of results want more parts (96 and more a row) than their list holds (2^20)."""
    from cosmokdtree_b200 import forest
    m, per = 300000, 8192
    P, Q = [], []
    for seed in (5, 6):
        rng = np.random.default_rng(seed)
        x = rng.normal(size=(m, 3))
        x *= 0.4 * rng.random((m, 1)) ** 2 / np.linalg.norm(x, axis=1, keepdims=True)
        P.append(x)
        Q.append(x[np.argsort((x * x).sum(1))[20000:20000 + per]])
    f = forest.build_forest(np.concatenate(P), [0, m, 2 * m], leaf=1)
    assert 66 < f.depth < 127
    return f, np.concatenate(Q), [0, per, 2 * per]


def test_gpu_cut_rows_boxes_past_the_part_list(gpu, core_forest):
    import torch
    from cosmokdtree_b200 import _lib
    f, q, qoff = core_forest
    Q = torch.from_numpy(q).cuda()
    B = torch.stack([Q - 0.003, Q + 0.003], 2).reshape(-1, 6).contiguous()
    o, idx = f.box_csr(B, qoff)
    assert int((o[1:] - o[:-1]).min()) >= 4096  # every row is long enough to be cut
    want, _ = whole(_lib.load(), _lib, f.handle, B, o, None, 0,
                    torch.tensor(qoff, device="cuda"))
    assert torch.equal(idx, want)


@pytest.mark.parametrize("sorted_", [0, 1])
def test_gpu_cut_rows_balls_past_the_part_list(gpu, core_forest, sorted_):
    """Warps that find the list full while others fill it walk their rows on."""
    import torch
    from cosmokdtree_b200 import _lib
    f, q, qoff = core_forest
    Q = torch.from_numpy(q).cuda()
    o, idx, dist = f.ball_csr(Q, qoff, 0.003, sorted=bool(sorted_))
    assert int((o[1:] - o[:-1]).min()) >= 4096
    wi, wd = whole(_lib.load(), _lib, f.handle, Q, o, 0.003, sorted_,
                   torch.tensor(qoff, device="cuda"))
    assert torch.equal(idx, wi) and torch.equal(dist, wd)


def test_gpu_cut_rows_end_where_the_offsets_say(gpu):
    """A fill with a larger radius than the count's truncates its rows, cut or whole."""
    import torch
    from cosmokdtree_b200 import _lib
    L = _lib.load()
    P = torch.from_numpy(cluster(1 << 19, 3, 3)).cuda()
    Q = P[(P * P).sum(1).argsort()[1000:1300]].contiguous()
    t = gpu.kdtree.build_kdtree(P)
    off, _, _ = gpu.kdtree.ball_search_csr(t, Q, 0.004)
    total, guard = int(off[-1]), 1 << 24
    assert total >= 192 * 300
    want, wd = whole(L, _lib, t.handle, Q, off, 0.005, 0)
    idx = torch.full((total + guard,), -7, dtype=torch.int64, device="cuda")
    dist = torch.full((total + guard,), -7.0, dtype=torch.float64, device="cuda")
    ptr = lambda x: ctypes.c_void_p(x.data_ptr())
    _lib.check(L.ckd_ball_fill_sized(t.handle, ptr(Q), 300, 0.005, 0, total, ptr(off), ptr(idx),
                                     ptr(dist), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
    assert bool((idx[total:] == -7).all()) and bool((dist[total:] == -7.0).all())
    assert torch.equal(idx[:total], want) and torch.equal(dist[:total], wd)
