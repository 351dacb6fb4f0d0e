"""Batches large enough to be sorted by default: k = 1 and 2 (a thread per query) and
longer lists (groups), on both sides of the lines of the rule and with the sort forced
on and off.  Every way gives the same rows, bit for bit, and a sample of them is the
model's."""
import numpy as np
import pytest

import spec

pytestmark = pytest.mark.gpu


def run(tree, q, k, md, bits):
    import torch
    tree.set_knn_bin_bits(bits)
    n = len(q)
    o = [torch.full((n, k), 7, dtype=torch.int32, device="cuda:0"), torch.full((n, k), 7.0, device="cuda:0"),
         torch.full((n, k, 3), 7.0, device="cuda:0"), torch.full((n,), 7, dtype=torch.int32, device="cuda:0")]
    torch.cuda.synchronize()
    tree.knn_device(q.data_ptr(), n, k, md, *(x.data_ptr() for x in o))
    tree.synchronize()
    return o


@pytest.mark.parametrize("kind", ["uniform", "lattice", "tiny"])
@pytest.mark.parametrize("nq", [899999, 900000, 1000033])
def test_every_way_gives_the_same_rows(ikdg_mod, kind, nq):
    import torch
    rng = np.random.default_rng(nq)
    n = 3 if kind == "tiny" else 30000
    pts = (rng.integers(0, 9, (n, 3)) if kind == "lattice" else rng.uniform(0, 9, (n, 3))).astype(np.float32)
    tree, ref = ikdg_mod.KDTree(0.9, 0.9, 0.5), spec.SpecTree(0.5)
    tree.Build(pts)
    ref.Build(pts)
    if n > 3:  # full buckets and holes
        add = pts[:9000] + np.float32(0 if kind == "lattice" else 0.125)
        tree.Add_Points(add, False)
        ref.Add_Points(add, False)
        box = np.array([[2, 2, 2, 4, 5, 6]], np.float32)
        assert tree.Delete_Point_Boxes(box) == ref.Delete_Point_Boxes(box)
    q = rng.uniform(-1, 10, (nq, 3)).astype(np.float32)
    q[::7] = np.round(q[::7])
    q[5::1000] = np.inf
    q[6::1000] = np.nan
    dq = torch.from_numpy(q).to("cuda:0")
    at = rng.choice(nq, 40)
    at = at[np.isfinite(q[at]).all(1)]
    for k in (1, 2, 3, 5):
        for md in (np.inf, 0.75):
            auto = run(tree, dq, k, md, -1)
            for bits in (0, 3, 16):
                for a, b in zip(auto, run(tree, dq, k, md, bits)):
                    assert torch.equal(a, b) or torch.equal(a.view(torch.int32), b.view(torch.int32)), (k, md, bits)
            rid, rd2 = ref.knn(q[at], k, md)
            assert np.array_equal(auto[0].cpu().numpy()[at], rid)
            assert np.array_equal(auto[1].cpu().numpy()[at].view(np.uint32), rd2.view(np.uint32))
            assert np.array_equal(auto[3].cpu().numpy(), (auto[0].cpu().numpy() >= 0).sum(1))
    tree.close()
