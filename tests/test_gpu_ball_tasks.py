"""Ball rows whose whole-subtree ranges need more emission tasks than the task buffer holds:
the slots that the first row past its end leaves empty hold no work."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_gpu_ball_more_emission_tasks_than_the_buffer_holds(gpu):
    import torch
    n, nq = 300000, 900  # 74 tasks of 4096 points a row: 66600 tasks against 65536
    rng = np.random.default_rng(3)
    P = torch.from_numpy(rng.random((n, 3))).cuda()
    Q = torch.from_numpy(rng.random((nq, 3))).cuda()
    t = gpu.kdtree.build_kdtree(P)
    from cosmokdtree_b200.kdtree import ball_search_csr
    for _ in range(2):
        off, idx, dist = ball_search_csr(t, Q, 2.0)  # every ball holds every point
        assert int(off[-1]) == n * nq
        idx, dist = idx.reshape(nq, n), dist.reshape(nq, n)
        assert torch.equal(idx[0].sort().values, torch.arange(n, device="cuda"))
        assert bool((idx == idx[0]).all())  # leaf order, the same in every row
        for r in (0, nq // 2, nq - 1):
            d = P[idx[r]] - Q[r]
            want = torch.sqrt((d[:, 0] * d[:, 0] + d[:, 1] * d[:, 1]) + d[:, 2] * d[:, 2])
            assert torch.equal(dist[r], want)
        del off, idx, dist
