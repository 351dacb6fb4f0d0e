"""Every traversal ends: its steps on nodes and on leaves are counted against one
cap, and reaching it is reported as an error.  The trees here are sound; the cap is
lowered below what a search needs, which takes the same way out as a damaged tree
without one."""
import numpy as np
import pytest

import spec

pytestmark = pytest.mark.gpu

N = 100000


def pair(ikdg_mod, monkeypatch, cap):
    pts = np.random.default_rng(3).uniform(-20, 20, (N, 3)).astype(np.float32)
    monkeypatch.setenv("IKDG_MAX_VISITS", str(cap))
    capped = ikdg_mod.KDTree()
    monkeypatch.delenv("IKDG_MAX_VISITS")
    capped.Build(pts)
    return capped, pts


# A search for one point within 1e-6 of a place without any passes five or so records
# on its way down and looks into at most the one or two buckets whose box holds the
# place: only steps on records can reach this cap.
@pytest.mark.parametrize("nq,k", [(1, 1), (1, 64), (33, 5), (3000, 16), (5000, 8), (1, 65)])
def test_knn_steps_on_records_count(ikdg_mod, monkeypatch, nq, k):
    tree, pts = pair(ikdg_mod, monkeypatch, 3)
    q = np.random.default_rng(4).uniform(-19, 19, (nq, 3)).astype(np.float32)
    with pytest.raises(ikdg_mod.IkdgError, match="loop cap") as e:
        tree.knn(q, k, 1e-6)
    assert e.value.status == ikdg_mod.INTERNAL
    tree.close()


def test_batch_and_range_searches_count(ikdg_mod, monkeypatch):
    import torch
    tree, pts = pair(ikdg_mod, monkeypatch, 3)
    q = np.random.default_rng(5).uniform(-19, 19, (64, 3)).astype(np.float32)
    dq = torch.from_numpy(q).to("cuda:0")
    ids = torch.empty((64, 4), dtype=torch.int32, device="cuda:0")
    d2 = torch.empty((64, 4), dtype=torch.float32, device="cuda:0")
    b = ikdg_mod.Batch()
    b.add_knn(tree, dq.data_ptr(), 64, 4, 1e-6, ids.data_ptr(), d2.data_ptr())
    torch.cuda.synchronize()
    b.run()
    with pytest.raises(ikdg_mod.IkdgError, match="loop cap"):
        b.synchronize()
    b.close()
    with pytest.raises(ikdg_mod.IkdgError, match="loop cap"):
        tree.radius_search(q, 1.0)
    with pytest.raises(ikdg_mod.IkdgError, match="loop cap"):
        tree.box_search(np.concatenate([q - 1, q + 1], 1))
    tree.close()


def test_write_pass_of_a_range_search_reports(ikdg_mod, monkeypatch):
    # The counting pass takes subtrees that the box covers as a whole, a handful of
    # steps; the write pass has every bucket to go through, 800 steps at the least.
    tree, pts = pair(ikdg_mod, monkeypatch, 400)
    box = np.array([[-30, -30, -30, 30, 30, 30]], np.float32)
    with pytest.raises(ikdg_mod.IkdgError, match="loop cap"):
        tree.box_search(box)
    with pytest.raises(ikdg_mod.IkdgError, match="loop cap"):
        tree.radius_search(np.zeros((1, 3), np.float32), 60.0)
    tree.close()


def test_default_cap_allows_the_longest_searches(ikdg_mod):
    # every point equally far: no subtree can be skipped, eight such queries a warp
    pts = np.full((20000, 3), 1.5, np.float32)
    tree, ref = ikdg_mod.KDTree(), spec.SpecTree()
    tree.Build(pts)
    ref.Build(pts)
    q = np.zeros((2056, 3), np.float32)
    ids, d2, _, _ = tree.knn(q, 5)
    rid, rd2 = ref.knn(q[:1], 5)
    assert (ids == rid).all() and (d2 == rd2).all()
    offs, ids, _ = tree.radius_search(q[:40], 10.0)
    assert (np.diff(offs) == len(pts)).all()
    tree.close()
