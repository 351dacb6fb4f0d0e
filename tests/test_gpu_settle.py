"""Mutations that end without a rebuild, with one job, with many jobs, with the
whole tree as the job, and with overflow points, on trees of one leaf up to more
leaves than the settling launch has threads.  The structure is validated and the
stored points equal the model's."""
import numpy as np
import pytest

import spec

pytestmark = pytest.mark.gpu


def same(tree, ref, rng):
    assert tree.validate() == 0 and tree.validnum() == ref.validnum()
    if ref.validnum() == 0:
        return
    q = rng.uniform(-55, 55, (12, 3)).astype(np.float32)
    ids, d2, _, _ = tree.knn(q, 6)
    rid, rd2 = ref.knn(q, 6)
    assert np.array_equal(ids, rid) and np.array_equal(d2, rd2)


@pytest.mark.parametrize("n", [1, 31, 33, 2000, 40000, 700001, 1060000])
def test_edit_sequences(ikdg_mod, n):
    rng = np.random.default_rng(n)
    pts = rng.uniform(-50, 50, (n, 3)).astype(np.float32)
    tree, ref = ikdg_mod.KDTree(0.3, 0.6, 0.5), spec.SpecTree(0.5)
    for t in (tree, ref):
        t.Build(pts)
    # one spot takes many points: full buckets overflow into a rebuild
    steps = [rng.uniform(49, 50, (600, 3)), rng.uniform(-50, 50, (3, 3)), rng.uniform(-50, 50, (n // 8 + 1, 3))]
    for add in steps:
        for t in (tree, ref):
            t.Add_Points(add.astype(np.float32), False)
        same(tree, ref, rng)
    # nothing hit; a few points; scattered slabs (many jobs); all that is left
    slabs = np.array([[x, -50, -50, x + 2.5, 50, 50] for x in range(-48, 48, 6)], np.float32)
    for boxes in (np.array([[60, 60, 60, 61, 61, 61]], np.float32), np.array([[0, 0, 0, 3, 3, 3]], np.float32), slabs,
                  np.array([[-60, -60, -60, 60, 60, 60]], np.float32)):
        assert tree.Delete_Point_Boxes(boxes) == ref.Delete_Point_Boxes(boxes)
        same(tree, ref, rng)
    for t in (tree, ref):
        t.Add_Points(pts[:100], False)
    tree.rebuild()
    same(tree, ref, rng)
    tree.close()


@pytest.mark.parametrize("hit", [1, 7, 400, 9000, 30000])
def test_refit_meetings(ikdg_mod, hit):
    """From one dirty bucket up to every bucket of the map: walks that meet at no
    node, at the upper nodes, at every node; twice on the same nodes."""
    rng = np.random.default_rng(hit)
    pts = rng.uniform(-50, 50, (30000, 3)).astype(np.float32)
    tree, ref = ikdg_mod.KDTree(0.9, 0.95, 0.5), spec.SpecTree(0.5)  # (nothing is rebuilt but full buckets)
    for t in (tree, ref):
        t.Build(pts)
    for seed in range(2):
        sel = rng.permutation(len(pts))[:hit]
        for t in (tree, ref):
            t.Delete_Points(pts[sel])
        same(tree, ref, rng)
        assert np.array_equal(np.asarray(tree.tree_range()).reshape(-1), ref.tree_range())
        for t in (tree, ref):
            t.Add_Points(pts[sel], False)
        same(tree, ref, rng)
    tree.close()


@pytest.mark.parametrize("n", [1, 5, 40, 300, 5000, 120000])
@pytest.mark.parametrize("dup", [False, True])
def test_box_and_point_deletion_walks(ikdg_mod, n, dup):
    """One to many boxes a call (the deletion splits the tree over more warps the fewer
    there are), covering all, touching faces, far off, overlapping; point deletions
    with several stored points within the match distance."""
    rng = np.random.default_rng(n)
    pts = rng.uniform(-50, 50, (n, 3)).astype(np.float32)
    if dup:
        pts[n // 2:] = pts[: n - n // 2]  # pairs of equal points
    tree, ref = ikdg_mod.KDTree(0.5, 0.6, 0.5), spec.SpecTree(0.5)
    for t in (tree, ref):
        t.Build(pts)
    lo = rng.uniform(-55, 50, (1500, 3))
    many = np.c_[lo, lo + rng.uniform(0, 4, (1500, 3))].astype(np.float32)
    face = np.r_[pts[0], pts[0] + 3][None].astype(np.float32)  # half-open: pts[0] is inside
    face2 = np.r_[pts[n // 3] - 3, pts[n // 3]][None].astype(np.float32)  # and outside here
    for boxes in (face, face2, many[:3], many[:130], many, np.array([[-60, -60, -60, 0, 60, 60]], np.float32)):
        assert tree.Delete_Point_Boxes(boxes) == ref.Delete_Point_Boxes(boxes)
        same(tree, ref, rng)
    for t in (tree, ref):
        t.Add_Points(pts[: n // 2], False)
    gone = np.r_[pts[:: max(1, n // 200)], pts[:3] + 3e-7, rng.uniform(-50, 50, (20, 3)).astype(np.float32)]
    for t in (tree, ref):
        t.Delete_Points(gone.astype(np.float32))
    assert tree.validate() == 0 and tree.validnum() == ref.validnum()
    every = np.array([[-60, -60, -60, 60, 60, 60]], np.float32)
    assert tree.Delete_Point_Boxes(every) == ref.Delete_Point_Boxes(every)
    assert tree.validnum() == 0 and tree.validate() == 0
    tree.close()


@pytest.mark.parametrize("spread", [0.05, 0.6, 6.0])
def test_voxel_search_teams(ikdg_mod, monkeypatch, spread):
    """Downsampling insertion where voxels hold many, a few and no stored points, with
    and without room for the pair list."""
    rng = np.random.default_rng(3)
    pts = rng.uniform(-4, 4, (9001, 3)).astype(np.float32)
    for cap in (None, "16"):
        if cap:
            monkeypatch.setenv("IKDG_DS_PAIR_CAP", cap)
        tree, ref = ikdg_mod.KDTree(0.5, 0.6, 0.5), spec.SpecTree(0.5)
        for t in (tree, ref):
            t.Build(pts)
        for seed in range(2):
            add = (rng.normal(0, spread, (301, 3))).astype(np.float32)
            assert tree.Add_Points(add, True) == ref.Add_Points(add, True)
            same(tree, ref, rng)
        tree.close()


@pytest.mark.parametrize("n", [400, 32768, 32769])
def test_voxel_groups_of_every_length(ikdg_mod, n):
    """New points at both hash widths of the grouper, voxels with 1 to 40 of them
    (folded by a thread or by a warp)."""
    rng = np.random.default_rng(n)
    reps = np.resize([1, 1, 2, 3, 15, 16, 17, 18, 33, 40], n)
    vox = np.repeat(np.arange(n), reps)[:n]
    corner = np.stack([vox % 37, vox // 37 % 41, vox // (37 * 41)], 1) * 0.5
    pts = (corner + rng.uniform(0.02, 0.48, (n, 3)))[rng.permutation(n)].astype(np.float32)
    tree, ref = ikdg_mod.KDTree(0.5, 0.6, 0.5), spec.SpecTree(0.5)
    base = rng.uniform(0, 20, (200, 3)).astype(np.float32)
    for t in (tree, ref):
        t.Build(base)
    assert tree.Add_Points(pts, True) == ref.Add_Points(pts, True)
    same(tree, ref, rng)
    xyz, ids = tree.flatten(with_ids=True)
    want, wid = ref.valid_points()
    assert np.array_equal(np.sort(ids), np.sort(wid))
    assert np.array_equal(xyz[np.argsort(ids)], want[np.argsort(wid)])
    tree.close()


def test_rebuild_jobs_of_a_large_map(ikdg_mod):
    """So many leaves and nodes that the jobs list what is below them.  Overflowing buckets, scattered jobs, one large job, the whole tree."""
    rng = np.random.default_rng(8)
    n = 2_900_000
    pts = rng.uniform(-50, 50, (n, 3)).astype(np.float32)
    tree, ref = ikdg_mod.KDTree(0.3, 0.6, 0.5), spec.SpecTree(0.5)
    for t in (tree, ref):
        t.Build(pts)
    spot = rng.uniform(10, 10.4, (3000, 3)).astype(np.float32)
    for t in (tree, ref):
        t.Add_Points(spot, False)
    same(tree, ref, rng)
    cubes = rng.uniform(-50, 47, (60, 3))
    for boxes in (np.c_[cubes, cubes + 3], np.array([[-50, -50, -50, -20, 50, 50]]), np.array([[0, 0, 0, 1e-3, 1, 1]])):
        boxes = boxes.astype(np.float32)
        assert tree.Delete_Point_Boxes(boxes) == ref.Delete_Point_Boxes(boxes)
        same(tree, ref, rng)
    tree.rebuild()
    same(tree, ref, rng)
    gone = tree.acquire_removed_points()
    assert len(gone) + tree.validnum() == n + len(spot)
    tree.close()
