"""Builds at the edges of the builder's paths (whole-block finish up to 4,096
points, multi-block splitter above) and on inputs
that make its selection long: lattices (many equal keys), all points equal, two
values, a far outlier that puts nearly every point into one bin.  The structure
is validated, the stored points are the input, and searches equal the model."""
import numpy as np
import pytest

import spec

pytestmark = pytest.mark.gpu

GEN = {
    "uniform": lambda rng, n: rng.uniform(-50, 50, (n, 3)),
    "lattice": lambda rng, n: rng.integers(0, 12, (n, 3)),
    "equal": lambda rng, n: np.full((n, 3), 3.5),
    "outlier": lambda rng, n: np.r_[rng.normal(0, 1, (n - 1, 3)), [[1e9, -1e9, 1e9]]],
    "two": lambda rng, n: np.c_[rng.integers(0, 2, (n, 2)), np.zeros(n)],
}


@pytest.mark.parametrize("kind", sorted(GEN))
@pytest.mark.parametrize("n", [4095, 4096, 4097, 8192, 8193, 32769, 65537, 140001])
def test_paths_and_degenerate_inputs(ikdg_mod, n, kind):
    rng = np.random.default_rng(n)
    pts = GEN[kind](rng, n).astype(np.float32)
    tree = ikdg_mod.KDTree(0.5, 0.6, 0.5)
    tree.Build(pts)
    for again in range(2):
        assert tree.validate() == 0
        xyz, ids = tree.flatten(with_ids=True)
        o = np.argsort(ids)
        assert np.array_equal(ids[o], np.arange(n)) and np.array_equal(xyz[o].view(np.uint32), pts.view(np.uint32))
        tree.rebuild()
    ref = spec.SpecTree(0.5)
    ref.Build(pts)
    q = np.concatenate([pts[:: n // 8][:8], rng.uniform(-2, 14, (8, 3)).astype(np.float32)])
    ids, d2, _, _ = tree.knn(q, 5)
    rid, rd2 = ref.knn(q, 5)
    assert np.array_equal(ids, rid) and np.array_equal(d2.view(np.uint32), rd2.view(np.uint32))
    tree.close()


def test_mixed_jobs_of_one_rebuild(ikdg_mod):
    """One mutation whose rebuild jobs take different paths: half of a large map
    deleted in stripes, small and large subtrees at once."""
    rng = np.random.default_rng(4)
    pts = rng.uniform(-50, 50, (300000, 3)).astype(np.float32)
    tree, ref = ikdg_mod.KDTree(0.3, 0.6, 0.5), spec.SpecTree(0.5)
    tree.Build(pts)
    ref.Build(pts)
    boxes = np.array([[-50, -50, -50, -10, 50, 50], [0, 0, 0, 6, 6, 6], [20, -40, -50, 24, -30, 50],
                      [30, 10, -50, 50, 14, 20]], np.float32)
    assert tree.Delete_Point_Boxes(boxes) == ref.Delete_Point_Boxes(boxes)
    assert tree.validate() == 0 and tree.validnum() == ref.validnum()
    add = rng.uniform(0, 3, (60000, 3)).astype(np.float32)
    tree.Add_Points(add, False)
    ref.Add_Points(add, False)
    assert tree.validate() == 0 and tree.validnum() == ref.validnum()
    q = rng.uniform(-50, 50, (16, 3)).astype(np.float32)
    ids, d2, _, _ = tree.knn(q, 9)
    rid, rd2 = ref.knn(q, 9)
    assert np.array_equal(ids, rid) and np.array_equal(d2, rd2)
    tree.close()
