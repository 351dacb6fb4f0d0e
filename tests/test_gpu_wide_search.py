"""kNN over the wide records at its edges: both group widths (batches below and
from 131,072 queries), every list size on both sides of a register boundary,
points on a lattice (whole shells of equal distances, ties by id), buckets with
more than the 16 slots of a leaf step, and trees whose leaves sit at any depth
inside a wide record.  Everything is bit-exact, so no tolerance appears."""
import numpy as np
import pytest

import spec

pytestmark = pytest.mark.gpu

KS = (1, 4, 5, 8, 9, 16, 17, 32, 33, 64)


def lattice(rng, n, cells):
    return rng.integers(0, cells, (n, 3)).astype(np.float32)


def check(tree, ref, q, k, md, reps=1):
    """The first rows against the model; with reps > 1 the batch is the same
    queries repeated, and every repeat must give the same rows."""
    rid, rd2 = ref.knn(q, k, md)
    ids, d2, xyz, cnt = tree.knn(np.tile(q, (reps, 1)), k, md)
    for r in range(reps):
        s = slice(r * len(q), (r + 1) * len(q))
        assert np.array_equal(ids[s], rid) and np.array_equal(d2[s].view(np.uint32), rd2.view(np.uint32)), (k, md, r)
        assert np.array_equal(cnt[s], (rid >= 0).sum(1))


@pytest.mark.parametrize("n", [1, 2, 17, 33, 65, 130, 257, 1100])
def test_lattice_ties_small_trees(ikdg_mod, n):
    rng = np.random.default_rng(n)
    for fill in (8, 16, 32):
        tree, ref = ikdg_mod.KDTree(), spec.SpecTree()
        tree.set_leaf_fill(fill)
        pts = lattice(rng, n, 6)
        tree.Build(pts)
        ref.Build(pts)
        q = lattice(rng, 130, 7) * np.float32(0.5)
        for k in KS:
            for md in (np.inf, 2.0):
                check(tree, ref, q, k, md)
        tree.close()


def test_both_group_widths(ikdg_mod):
    rng = np.random.default_rng(5)
    tree, ref = ikdg_mod.KDTree(0.5, 0.6, 0.5), spec.SpecTree(0.5)
    pts = lattice(rng, 6000, 12)
    tree.Build(pts)
    ref.Build(pts)
    # appended points fill buckets past 16 slots, a deletion leaves holes
    add = lattice(rng, 3000, 12)
    tree.Add_Points(add, False)
    ref.Add_Points(add, False)
    box = np.array([[2, 2, 2, 6, 7, 8]], np.float32)
    assert tree.Delete_Point_Boxes(box) == ref.Delete_Point_Boxes(box)
    assert tree.validate() == 0
    q = rng.uniform(-1, 13, (1024, 3)).astype(np.float32)
    q[:300] = lattice(rng, 300, 12)
    for k in KS:
        check(tree, ref, q, k, np.inf)
        check(tree, ref, q, k, 1.5, reps=129)  # 132,096 queries
    tree.close()
