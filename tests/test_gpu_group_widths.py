"""kNN at the line between a warp per query and eight queries a warp (2,048 queries),
with last blocks that are partly filled, for list sizes on both sides of the register
steps: into ordinary host arrays, into page-locked ones that start off a 16-byte
boundary, and on the device.  All ways and the model agree bit for bit."""
import numpy as np
import pytest

import spec

pytestmark = pytest.mark.gpu

KS = (1, 4, 5, 8, 9, 16, 17, 32, 33, 64)


@pytest.mark.parametrize("nq", [1, 5, 31, 33, 2047, 2048, 2049, 2083, 4097])
def test_all_buffers(ikdg_mod, nq):
    import torch
    rng = np.random.default_rng(nq)
    pts = rng.uniform(-8, 8, (20000, 3)).astype(np.float32)
    tree, ref = ikdg_mod.KDTree(), spec.SpecTree()
    tree.Build(pts)
    ref.Build(pts)
    q = rng.uniform(-9, 9, (nq, 3)).astype(np.float32)
    dq = torch.from_numpy(q).to("cuda:0")
    sample = rng.choice(nq, min(nq, 24), replace=False)
    for k in KS:
        for md in (np.inf, 0.9):
            want = tree.knn(q, k, md)
            rid, rd2 = ref.knn(q[sample], k, md)
            assert np.array_equal(want[0][sample], rid)
            assert np.array_equal(want[1][sample].view(np.uint32), rd2.view(np.uint32))
            assert np.array_equal(want[3], (want[0] >= 0).sum(1))
            rows = nq * k
            # page-locked, every array 4, 8 or 12 bytes off
            for off in (1, 2, 3):
                buf = torch.full((5 * rows + nq + 16 + 3 * nq + 16,), -5.0, pin_memory=True).numpy()
                at, out = off, []
                for n, t, s in ((rows, np.int32, (nq, k)), (rows, np.float32, (nq, k)), (3 * rows, np.float32, (nq, k, 3)),
                                (nq, np.int32, (nq,))):
                    out.append(buf[at:at + n].view(t).reshape(s))
                    at += n + (1 if off == 2 else 0)
                pq = buf[at + 1:at + 1 + 3 * nq].reshape(nq, 3)
                pq[:] = q
                tree.knn_into(pq.ctypes.data, nq, k, md, *(o.ctypes.data for o in out))
                for a, b in zip(out, want):
                    assert np.array_equal(a, b), (k, md, off)
                assert (buf[:off] == -5.0).all() and buf[at] == -5.0
            dev = [torch.empty(o.shape, dtype=torch.int32 if o.dtype == np.int32 else torch.float32, device="cuda:0")
                   for o in want]
            torch.cuda.synchronize()
            tree.knn_device(dq.data_ptr(), nq, k, md, *(d.data_ptr() for d in dev))
            tree.synchronize()
            for a, b in zip(dev, want):
                assert np.array_equal(a.cpu().numpy(), b), (k, md, "device")
    tree.close()
