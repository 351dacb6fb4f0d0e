"""A rebuild that finds no room ends with an error and leaves the tree as it was: it
answers as before, can be changed, and a rebuild that fits goes through."""
import numpy as np
import pytest

import spec

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [9000, 60000])  # the root at different places of the top record
def test_tree_survives(ikdg_mod, monkeypatch, n):
    rng = np.random.default_rng(n)
    pts = rng.uniform(-10, 10, (n, 3)).astype(np.float32)
    # A build of n points reserves n / 8 leaves and a quarter more; the first rebuild
    # wants as many again beside those in use.
    monkeypatch.setenv("IKDG_POOL_LIMIT", str(int(0.19 * n)))
    tree = ikdg_mod.KDTree(0.5, 0.6, 0.5)
    monkeypatch.delenv("IKDG_POOL_LIMIT")
    ref = spec.SpecTree(0.5)
    tree.Build(pts)
    ref.Build(pts)
    q = rng.uniform(-10, 10, (60, 3)).astype(np.float32)

    def same():
        for k in (1, 8, 65):
            ids, d2, _, _ = tree.knn(q, k)
            rid, rd2 = ref.knn(q, k)
            assert np.array_equal(ids, rid) and np.array_equal(d2.view(np.uint32), rd2.view(np.uint32))
        assert tree.validate() == 0 and tree.validnum() == ref.validnum()

    same()
    with pytest.raises(ikdg_mod.IkdgError) as e:
        tree.rebuild()
    assert e.value.status == ikdg_mod.CAPACITY
    same()
    # small jobs still fit, and are sized afresh
    box = np.array([[-1, -1, -1, 1, 1.5, 1]], np.float32)
    assert tree.Delete_Point_Boxes(box) == ref.Delete_Point_Boxes(box)
    same()
    # few enough points left: the whole tree can be rebuilt
    box = np.array([[-10, -10, -10, 10, 10, 6]], np.float32)
    assert tree.Delete_Point_Boxes(box) == ref.Delete_Point_Boxes(box)
    tree.rebuild()
    same()
    tree.close()
