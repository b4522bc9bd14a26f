"""The dilation loop's step limits (W + H + D, or max_iterations) where several
steps run per barrier: pairs that are done just below the limit among pairs that
need many more steps."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

KEYS = ("hd", "hd_ab", "hd_ba", "sum_ab", "sum_ba", "n_a", "n_b", "n_a_not_b", "n_b_not_a", "status")


def corners(shape):
    """One voxel in opposite corners: the longest distance of the volume."""
    a, b = np.zeros(shape, np.uint8), np.zeros(shape, np.uint8)
    a[0, 0, 0] = b[-1, -1, -1] = 1
    return a, b


SHORT = [(1, 1, n) for n in range(2, 14)] + [(2, 2, 2), (2, 3, 4), (3, 3, 5), (1, 4, 4), (5, 6, 7), (8, 9, 10), (33, 2, 35)]


def _cuda(p):
    return tuple(torch.from_numpy(m).cuda() for m in p)


@pytest.mark.parametrize("metric", ["se6", "se18"])
@pytest.mark.parametrize("steps", [1, 2, 3, 4, 5])
def test_short_pairs_beside_a_long_one(hd, oracle, metric, steps):
    pairs = [corners(s) for s in SHORT] + [corners((40, 50, 60))]
    with hd.Context(0, kernel=2, steps_per_barrier=steps) as c:
        for i, (r, p) in enumerate(zip(c.batch([_cuda(p) for p in pairs], metric), pairs)):
            o = oracle.bfs_pair(*p, metric)
            assert all(r[k] == o[k] for k in KEYS), (i, r, o)


@pytest.mark.parametrize("metric,opts", [("se18", {}), ("se6", {"kernel": 2})])
def test_short_pairs_join_a_long_one(hd, oracle, metric, opts):
    """The server's shape for few requests runs 4 steps per barrier."""
    pairs = [corners(s) for s in SHORT]
    far = corners((200, 200, 200))
    dev, dfar = [_cuda(p) for p in pairs], _cuda(far)
    want, wfar = [oracle.bfs_pair(*p, metric) for p in pairs], None
    with hd.Context(0, **opts) as c, hd.Server(c, metric=metric) as srv:
        wfar = c.compute(*dfar, metric)
        for i, p in enumerate(dev):
            tf, t = srv.submit(*dfar), srv.submit(*p)
            r, rf = srv.wait(t, 60000), srv.wait(tf, 60000)
            assert all(r[k] == want[i][k] for k in KEYS), (i, r, want[i])
            assert all(rf[k] == wfar[k] for k in KEYS), (i, rf, wfar)


def test_hits_past_a_cap_on_the_steps(hd):
    """With 4 steps per barrier and at most 5 steps the second iteration runs to step
    8: B's voxels at distance 7 are counted, and A's counts (2 voxels at distance 5,
    which set the robust HD) stay their own."""
    a = torch.zeros((1, 40, 200), dtype=torch.uint8, device="cuda")
    a[:, 10:30, 50:150] = 1
    b = a.clone()
    a[:, 20:22, 154] = 1
    b[:, 30:33, 50:150] = 1
    b[:, 36, 100:105] = 1
    with hd.Context(0, kernel=2, steps_per_barrier=4) as c:
        want = c.compute(a, b, "se6")
    assert (want["hd_ab"], want["hd_ba"], want["hd_robust"]) == (5, 7, 5)
    with hd.Context(0, kernel=2, steps_per_barrier=4, max_iterations=5) as c:
        for r in [c.compute(a, b, "se6")] + c.batch([(a, b)] * 3, "se6"):
            assert all(r[k] == want[k] for k in KEYS + ("hd_robust", "avg_hd")), (r, want)
