"""kNN where many points coincide: buckets full of points as far as the k-th, of which
the smaller ids enter.  Places with fewer and more points than k, a bucket and a step
hold, deleted ones among them, and distance limits on, below and above the ties."""
import numpy as np
import pytest

import spec

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("places,each", [(1, 700), (3, 40), (40, 17), (300, 5), (27, 150)])
def test_ids_decide(ikdg_mod, places, each):
    rng = np.random.default_rng(places * each)
    site = rng.integers(0, 4, (places, 3)).astype(np.float32)
    n = places * each
    pts = site[rng.permutation(n) % places]
    tree, ref = ikdg_mod.KDTree(0.9, 0.9, 0.5), spec.SpecTree(0.5)
    tree.Build(pts)
    ref.Build(pts)
    add = site[rng.integers(0, places, n // 3)]
    q = np.concatenate([site[rng.integers(0, places, 37)], rng.integers(0, 5, (20, 3)).astype(np.float32),
                        rng.uniform(-1, 5, (16, 3)).astype(np.float32)])
    for step in range(2):
        for k in (1, 2, 4, 5, 8, 9, 16, 17, 32, 33, 64, 65):
            for md in (np.inf, 0.0, 1.0, np.sqrt(2.0)):
                ids, d2, _, _ = tree.knn(np.tile(q, (1 if k > 9 else 30, 1)), k, md)
                rid, rd2 = ref.knn(q, k, md)
                for at in range(0, len(ids), len(q)):
                    assert np.array_equal(ids[at:at + len(q)], rid), (k, md)
                    assert np.array_equal(d2[at:at + len(q)].view(np.uint32), rd2.view(np.uint32)), (k, md)
        if step == 0:
            tree.Add_Points(add, False)
            ref.Add_Points(add, False)
            # (which of several points at one place goes is not said, so boxes)
            lo = site[0] - np.float32(0.25)
            box = np.concatenate([lo, lo + np.float32(0.5)])[None]
            assert tree.Delete_Point_Boxes(box) == ref.Delete_Point_Boxes(box)
    tree.close()
