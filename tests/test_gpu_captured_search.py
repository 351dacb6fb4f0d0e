"""Device searches captured into a CUDA graph and replayed after mutations that did not
grow the tree's pools (a graph holds their addresses; here the pools have grown before):
they answer like a call made then, although the root is another node and the tree has
other levels."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N = 60000


@pytest.mark.parametrize("before,after", [(16, 16), (32, 8), (8, 32), (8, 16)])
def test_replay_after_rebuilds(ikdg_mod, monkeypatch, before, after):
    import torch
    # (no validation between calls: it adds nothing here)
    monkeypatch.delenv("IKDG_DEBUG_VALIDATE", raising=False)
    rng = np.random.default_rng(before + after)
    pts = rng.uniform(-10, 10, (N, 3)).astype(np.float32)
    tree = ikdg_mod.KDTree(0.9, 0.95, 0.5)
    # room for leaves of eight points and more: later rebuilds need less
    tree.set_leaf_fill(8)
    tree.Build(pts)
    for _ in range(3):
        tree.rebuild()
    tree.set_leaf_fill(before)
    tree.rebuild()

    dev = "cuda:0"
    q = torch.from_numpy(rng.uniform(-10, 10, (3000, 3)).astype(np.float32)).to(dev)
    r = torch.full((3000,), 0.6, device=dev)
    box = torch.cat([q - 0.5, q + 0.5], 1).contiguous()
    cap = 400000
    knn = {k: (torch.empty((3000, k), dtype=torch.int32, device=dev), torch.empty((3000, k), device=dev)) for k in (1, 9, 40)}
    na = (torch.empty((3000, 5), dtype=torch.int32, device=dev), torch.empty((3000, 5), device=dev))
    rng_out = [(torch.zeros(3001, dtype=torch.int64, device=dev), torch.zeros(cap, dtype=torch.int32, device=dev))
               for _ in range(2)]

    def search():
        for k, (i, d) in knn.items():
            tree.knn_device(q.data_ptr(), 3000, k, np.inf, i.data_ptr(), d.data_ptr())
        tree.knn_device_noalloc(q.data_ptr(), 3000, 5, np.inf, na[0].data_ptr(), na[1].data_ptr())
        tree.radius_search_device(q.data_ptr(), 3000, r.data_ptr(), rng_out[0][0].data_ptr(), rng_out[0][1].data_ptr(), cap)
        tree.box_search_device(box.data_ptr(), 3000, rng_out[1][0].data_ptr(), rng_out[1][1].data_ptr(), cap)

    def results():
        torch.cuda.synchronize()
        out = [t.cpu().numpy().copy() for pair in list(knn.values()) + [na] for t in pair]
        for offs, ids in rng_out:
            offs, ids = offs.cpu().numpy(), ids.cpu().numpy()
            assert offs[-1] <= cap
            out += [offs.copy()] + [np.sort(ids[a:b]) for a, b in zip(offs[:-1], offs[1:])]
        return out

    torch.cuda.synchronize()
    search()  # the arenas have their size
    tree.synchronize()
    graph = torch.cuda.CUDAGraph()
    stream = torch.cuda.ExternalStream(tree.stream())
    with torch.cuda.stream(stream):
        graph.capture_begin(capture_error_mode="thread_local")
        search()
        graph.capture_end()
    for step in range(3):
        if step == 1:
            tree.Delete_Point_Boxes(np.array([[-10, -10, -10, 0, 0, 10]], np.float32))
        if step == 2:
            tree.set_leaf_fill(after)
        if step:
            tree.rebuild()
        for _, ids in rng_out:
            ids.zero_()
        torch.cuda.synchronize()
        with torch.cuda.stream(stream):
            graph.replay()
        got = results()
        search()
        want = results()
        assert len(got) == len(want) and all(np.array_equal(a, b) for a, b in zip(got, want)), step
    del graph
    tree.close()
