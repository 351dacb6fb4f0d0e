"""A tree with more levels than the searches' stacks are sized for: every search and
every batch run says so and returns.  (The height guard keeps real trees far below; the
limit is lowered here.)"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def small_limit_tree(ikdg_mod, monkeypatch, levels):
    monkeypatch.setenv("IKDG_MAX_LEVELS", str(levels))
    t = ikdg_mod.KDTree(0.5, 0.6, 0.5)
    monkeypatch.delenv("IKDG_MAX_LEVELS")
    return t


def test_searches_refuse_and_the_batch_run_returns(ikdg_mod, monkeypatch):
    import torch
    rng = np.random.default_rng(2)
    tree = small_limit_tree(ikdg_mod, monkeypatch, 8)
    pts = rng.uniform(-10, 10, (100000, 3)).astype(np.float32)
    tree.Build(pts[:1500])  # 7 levels at most
    q = rng.uniform(-10, 10, (16, 3)).astype(np.float32)
    dq = torch.from_numpy(q).to("cuda:0")
    ids = torch.empty((16, 4), dtype=torch.int32, device="cuda:0")
    d2 = torch.empty((16, 4), dtype=torch.float32, device="cuda:0")
    b = ikdg_mod.Batch()
    b.add_knn(tree, dq.data_ptr(), 16, 4, np.inf, ids.data_ptr(), d2.data_ptr())
    torch.cuda.synchronize()
    b.run()
    b.synchronize()
    want = tree.knn(q, 4)
    assert np.array_equal(ids.cpu().numpy(), want[0])
    tree.Build(pts)  # 13 levels: above the limit, and above the batch's plan
    deeper = dict(match="deeper than")
    with pytest.raises(ikdg_mod.IkdgError, **deeper):
        b.run()
    for call in (lambda: tree.knn(q, 4), lambda: tree.knn(np.tile(q, (300, 1)), 4), lambda: tree.knn(q, 70),
                 lambda: tree.radius_search(q, 1.0), lambda: tree.box_search(np.concatenate([q, q + 1], 1)),
                 lambda: tree.knn_device(dq.data_ptr(), 16, 4, np.inf, ids.data_ptr(), d2.data_ptr()),
                 lambda: tree.knn_device_noalloc(dq.data_ptr(), 16, 4, np.inf, ids.data_ptr(), d2.data_ptr())):
        with pytest.raises(ikdg_mod.IkdgError, **deeper):
            call()
    tree.Build(pts[:1500])
    b.run()
    b.synchronize()
    assert np.array_equal(ids.cpu().numpy(), want[0])
    b.close()
    tree.close()
