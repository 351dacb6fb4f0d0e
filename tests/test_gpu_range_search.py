"""Box and radius search at the edges of the warp-per-queries kernels: batches on
both sides of every queries-per-warp step, searches with no hits, one point, all
points (covered subtrees counted as a whole, whose hits are then searched again
instead of read from the hit log), buckets with more than 16 slots, capacities
that leave queries out.  Hit sets and offsets are compared exactly."""
import numpy as np
import pytest

import spec

pytestmark = pytest.mark.gpu


def build(ikdg_mod, rng, n, fill):
    tree, ref = ikdg_mod.KDTree(0.5, 0.6, 0.5), spec.SpecTree(0.5)
    tree.set_leaf_fill(fill)
    pts = rng.integers(-20, 21, (n, 3)).astype(np.float32) * np.float32(0.5)
    tree.Build(pts)
    ref.Build(pts)
    add = rng.uniform(-10, 10, (n // 3 + 1, 3)).astype(np.float32)
    tree.Add_Points(add, False)
    ref.Add_Points(add, False)
    hole = np.array([[-3, -3, -3, 1, 2, 4]], np.float32)
    assert tree.Delete_Point_Boxes(hole) == ref.Delete_Point_Boxes(hole)
    return tree, ref


def queries(rng, n):
    c = rng.uniform(-11, 11, (n, 3))
    s = rng.choice([0.0, 0.4, 2.0, 7.0, 60.0], (n, 1)) * rng.uniform(0.5, 1.0, (n, 3))
    return (np.concatenate([c - s / 2, c + s / 2], 1).astype(np.float32), c.astype(np.float32),
            (s[:, 0] / 2).astype(np.float32))


@pytest.mark.parametrize("n,fill", [(1, 16), (40, 8), (900, 16), (900, 32), (12000, 16)])
def test_hits_and_order(ikdg_mod, n, fill):
    rng = np.random.default_rng(n + fill)
    tree, ref = build(ikdg_mod, rng, n, fill)
    boxes, centres, radii = queries(rng, 150)
    for name, search, want in (("box", lambda k: tree.box_search(np.tile(boxes, (k, 1))), ref.box_search(boxes)),
                               ("radius", lambda k: tree.radius_search(np.tile(centres, (k, 1)), np.tile(radii, k)),
                                ref.radius_search(centres, radii))):
        first = None
        for k in (1, 66, 132):  # one, two and four queries a warp
            offs, ids, xyz = search(k)
            assert len(offs) == 150 * k + 1
            if first is None:
                first = (offs, ids, xyz)
                for i, w in enumerate(want):
                    assert np.array_equal(np.sort(ids[offs[i]:offs[i + 1]]), w), (name, i)
                pts = dict(zip(ref.valid_points()[1].tolist(), ref.valid_points()[0]))
                for j in range(0, len(ids), 97):
                    assert np.array_equal(xyz[j], pts[int(ids[j])])
            else:  # every repeat gives the same hits in the same order
                assert np.array_equal(np.diff(offs), np.tile(np.diff(first[0]), k))
                assert np.array_equal(ids, np.tile(first[1], k)) and np.array_equal(xyz, np.tile(first[2], (k, 1)))
    tree.close()


def test_capacity_leaves_queries_out(ikdg_mod):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(9)
    tree, ref = build(ikdg_mod, rng, 5000, 16)
    boxes, _, _ = queries(rng, 10000)
    offs, ids, _ = tree.box_search(boxes)
    dev = torch.device("cuda")
    b = torch.from_numpy(boxes).to(dev)
    for cap in (0, int(offs[5000]) - 3, int(offs[-1])):
        o = torch.full((len(boxes) + 1,), -1, dtype=torch.int64, device=dev)
        out = torch.full((int(offs[-1]) + 1,), -7, dtype=torch.int32, device=dev)
        total = torch.zeros((1,), dtype=torch.int64, device=dev)
        torch.cuda.synchronize()
        tree.box_search_device(b.data_ptr(), len(boxes), o.data_ptr(), out.data_ptr(), cap, 0, total.data_ptr())
        torch.cuda.synchronize()
        assert np.array_equal(o.cpu().numpy(), offs) and int(total.item()) == offs[-1]
        got = out.cpu().numpy()
        fits = offs[1:] <= cap
        for i in range(0, len(boxes), 7):
            s = slice(offs[i], offs[i + 1])
            assert np.array_equal(got[s], ids[s] if fits[i] else np.full(offs[i + 1] - offs[i], -7)), i
    tree.close()
