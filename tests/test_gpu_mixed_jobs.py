"""One mutation with a large rebuild job, middle ones and many small ones: the large
splitter's levels hold segments of every size at once, listed by the jobs and by the
levels before.  The tree is validated, and its points and answers are those of the
points that were left."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,big,middle,small", [(300000, 0.25, 0, 1200), (1000000, 0.25, 6, 900), (1000000, 0.0, 40, 0)])
def test_jobs_of_every_size_in_one_call(ikdg_mod, n, big, middle, small):
    rng = np.random.default_rng(n + middle)
    pts = rng.uniform(-50, 50, (n, 3)).astype(np.float32)
    tree = ikdg_mod.KDTree(0.2, 0.6, 0.5)  # a fifth deleted: rebuild
    tree.Build(pts)
    boxes = [[-50, -50, -50, 0, -50 + 104 * big, 50]] if big else []
    # middle jobs: some 8,000 points each; small ones some 100
    for count, points in ((middle, 8000), (small, 100)):
        side = 100 * (points / n) ** (1 / 3)
        c = rng.uniform([2, -49, -49], 49 - side, (count, 3))
        boxes += list(np.concatenate([c, c + side], 1))
    b = np.array(boxes, np.float32)
    gone = np.zeros(n, bool)
    by_x = np.argsort(pts[:, 0])
    xs = pts[by_x, 0]
    for x in b:
        i = by_x[np.searchsorted(xs, x[0]):np.searchsorted(xs, x[3])]
        p = pts[i]
        gone[i[((p >= x[:3]) & (p < x[3:])).all(1)]] = True
    assert tree.Delete_Point_Boxes(b) == gone.sum()
    assert tree.validate() == 0 and tree.validnum() == n - gone.sum()
    xyz, ids = tree.flatten(with_ids=True)
    o = np.argsort(ids)
    assert np.array_equal(ids[o], np.flatnonzero(~gone))
    assert np.array_equal(xyz[o].view(np.uint32), pts[~gone].view(np.uint32))
    left = np.flatnonzero(~gone)
    q = rng.uniform(-50, 50, (12, 3)).astype(np.float32)
    got = tree.knn(q, 7)[0]
    for i in range(len(q)):
        d = (q[i] - pts[left]).astype(np.float32) ** 2
        d = (d[:, 0] + d[:, 1]) + d[:, 2]
        assert np.array_equal(got[i], left[np.lexsort((left, d))[:7]])
    tree.close()
